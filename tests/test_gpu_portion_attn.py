"""Prompt attention on tcgen05 against 64-bit softmax attention: page sizes (the boxes that fetch keys shrink with them), kept first keys
around box and tile edges, portions around the query and key tiles, several items per CTA, caches whose unused rows hold NaN, heads per
key head, value heads, float outputs, gates and caps."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64
LOST = [0]                                            # waits that ran out on purpose


@pytest.fixture(scope="module")
def nat():
    import nano_qwen3tts_vllm_b200._native as n
    n.lib()
    LOST[0] = n.portion_attn_timeouts()
    return n


class _Takes:
    """A call that this kernel takes, or leaves to another one; none of its waits may run out."""

    def __init__(self, nat, takes=True):
        self.nat, self.takes = nat, takes

    def __enter__(self):
        self.before = self.nat.portion_attn_launches()

    def __exit__(self, *exc):
        torch.cuda.synchronize()
        if exc[0] is None:
            assert self.nat.portion_attn_launches() - self.before == int(self.takes)
            assert self.nat.portion_attn_timeouts() == LOST[0]


def _case(nat, seqs, *, H=4, G=2, Gv=None, d=64, dv=64, page=16, kind="window", mask=0, keep=0, cap=0.0, sink=True, gate="head", scale=None,
          f32=False, seed=0, poison=False, known=False):
    """``seqs`` = [(cached, new)].  Everything in the caches that no sequence owns is NaN."""
    from tests.lm_util import Lay
    Gv = Gv or G
    g = torch.Generator().manual_seed(seed)
    need = [-(-(c + n) // page) for c, n in seqs]
    perm = (torch.randperm(sum(need), generator=g) + 1).tolist()
    tabs = [perm[sum(need[:i]):sum(need[:i + 1])] for i in range(len(need))]
    lay = Lay([(c, n, t) for (c, n), t in zip(seqs, tabs)], page, max(need))
    if known:
        lay.max_keys = max(c + n for c, n in seqs)
    r = lambda *s: torch.randn(s, generator=g)
    kc, vc = torch.full((sum(need) + 2, page, G * d), math.nan), torch.full((sum(need) + 2, page, Gv * dv), math.nan)
    n_tok = lay.n_tokens
    q, scale = r(n_tok, H * d).to(BF), scale if scale is not None else d ** -0.5
    sk, gt = r(H), r(n_tok, H * dv if gate == "element" else H).to(BF)
    ref, o = [], 0
    for (c, n), t in zip(seqs, tabs):
        k, v = r(c + n, G, d).to(BF), r(c + n, Gv, dv).to(BF)
        for p in range(c + n):
            kc[t[p // page], p % page], vc[t[p // page], p % page] = k[p].reshape(-1).float(), v[p].reshape(-1).float()
        i, j = torch.arange(c, c + n)[:, None], torch.arange(c + n)[None]
        ok = j <= i
        if mask:
            ok = ok & (((i - j < mask) if kind == "window" else (i // mask == j // mask)) | (j < keep))
        if poison:                                                   # values that no new token of the sequence sees
            for p in (~ok.any(0)).nonzero().flatten().tolist():
                vc[t[p // page], p % page], v[p] = math.inf, 0
        qq, out = q[o:o + n].view(n, H, d).to(F64), []
        for h in range(H):
            kg = h // (H // G)
            s = qq[:, h] @ k[:, kg].to(F64).T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~ok, -math.inf)
            if sink:
                s = torch.cat([s, sk[h].to(F64).expand(n, 1)], 1)
            p = s.softmax(-1)[:, :c + n]
            out.append(p @ v[:, kg % Gv].to(F64))
        y = torch.stack(out, 1)
        gg = torch.sigmoid(gt[o:o + n].to(F64))
        y = y * (gg.view(n, H, dv) if gate == "element" else gg[:, :, None] if gate == "head" else 1.0)
        ref.append(y.reshape(n, -1))
        o += n
    ref = torch.cat(ref)
    out = torch.empty(n_tok, H * dv, dtype=torch.float32 if f32 else BF, device=DEV)
    # the longest portion's keys up to which the other kernel is the faster one, where they are known
    short = 64 if cap == 0 and gate != "element" and H * lay.n_seqs <= 296 else 40
    with _Takes(nat, not known or lay.max_keys > short):
        nat.sink_attn(q.to(DEV), kc.to(BF).to(DEV), vc.to(BF).to(DEV), out, lay, sk.to(DEV) if sink else None, gt.to(DEV) if gate else None, H, G, d, dv,
                      page, nat.MASK_WINDOW if kind == "window" else nat.MASK_CHUNK, mask, scale, nat.SINK_ATTN_TENSOR, v_heads=Gv, keep_first=keep,
                      softcap=cap, gate_el=gate == "element")
    err = (out.double().cpu() - ref).abs().max() / ref.abs().max()
    # weights carry 16 bits and scores float sums (a few 1e-5 together); bf16 outputs round to 2^-9
    assert err.item() < (5e-5 if f32 else 4e-3), err.item()


@pytest.mark.parametrize("page", [16, 32, 48, 80, 256])
def test_page_sizes(nat, page):
    _case(nat, [(0, 150), (37, 141), (260, 5)], page=page, mask=70, seed=page, f32=True)


@pytest.mark.parametrize("keep", [1, 4, 15, 16, 17, 40, 127, 128, 129, 300])
@pytest.mark.parametrize("mask", [9, 130])
def test_kept_first_keys(nat, keep, mask):
    _case(nat, [(0, 200), (150, 90), (keep + mask - 1, 40), (keep + 20, 33)], mask=mask, keep=keep, seed=keep + mask, f32=True, sink=False, gate=None)


@pytest.mark.parametrize("H,G", [(2, 2), (4, 2), (6, 2), (8, 2), (16, 1), (5, 1)])
@pytest.mark.parametrize("d,dv", [(64, 64), (64, 128), (128, 64), (128, 128)])
def test_heads_per_key_head_and_sizes(nat, H, G, d, dv):
    _case(nat, [(0, 63), (3, 64), (0, 65), (500, 130), (8, 2), (11, 1)], H=H, G=G, d=d, dv=dv, mask=200, kind="chunk", gate="element", seed=H * d)


@pytest.mark.parametrize("n", [2, 127, 128, 129, 255, 257, 513])
@pytest.mark.parametrize("cached", [0, 1, 127, 128, 1000])
def test_portions_around_the_tiles(nat, n, cached):
    _case(nat, [(cached, n)], H=2, G=2, d=64, dv=64, page=64, seed=n + cached, cap=20.0 if n % 2 else 0.0, f32=n % 3 == 0)


def test_value_heads_shared_by_key_heads_and_negative_scale(nat):
    _case(nat, [(0, 140), (77, 60)], H=8, G=4, Gv=2, d=64, dv=128, mask=50, keep=3, sink=False, gate=None, f32=True)
    _case(nat, [(0, 140), (77, 60)], H=4, G=2, scale=-0.2, f32=True)


def test_scores_that_grow_along_the_keys(nat):
    """The running maximum moves in every tile: weights are rescaled again and again."""
    _case(nat, [(0, 700)], H=2, G=1, d=64, dv=64, scale=9.0, f32=True)


@pytest.mark.parametrize("n", [1500, 3001])
def test_several_items_for_every_cta(nat, n):
    """Two row tiles an item and more items than multiprocessors; the ring and its barriers go on from item to item."""
    _case(nat, [(0, n), (300, n - 700), (0, 1), (5, 33)], H=16, G=8, d=128, dv=128, page=64, mask=200, keep=4, gate="element", seed=n)


@pytest.mark.parametrize("seqs", [[(0, 300)] + [(50, 1)] * 40, [(30, 1)] * 33 + [(100, 257), (0, 65)], [(5, 33)] * 40, [(0, 128)] * 8 + [(9, 65), (0, 65)],
                                  [(300, 200)] * 6, [(50, 1)] * 240 + [(0, 130), (70, 400)]])
def test_portions_beside_decoded_tokens(nat, seqs):
    """One or two row tiles an item, by how many single ones (64 tokens of 2 of 16 heads) the portions really have: 40, 56, 160 and 80 take one, 320 and
    192 long ones two, where there are 148 multiprocessors.  Their longest portion, taken for all, says two everywhere, and
    more CTAs than multiprocessors in the last step."""
    _case(nat, seqs, H=16, G=8, d=128, dv=128, page=64, mask=100, keep=3, gate="head", seed=len(seqs))
    _sigmoid_case(nat, seqs, 16, 8, 128, 120, page=64)


def test_values_nobody_sees_may_be_infinite(nat):
    """Rows in front of the window, behind the last key and beyond the kept ones share tiles with visible rows."""
    _case(nat, [(700, 150), (90, 60)], H=4, G=2, d=64, dv=64, page=64, mask=100, keep=5, poison=True, f32=True)


@pytest.mark.parametrize("keys", [2, 39, 40, 41, 64, 65])
@pytest.mark.parametrize("gate,cap,more", [("element", 0.0, 0), ("head", 0.0, 0), (None, 20.0, 0), (None, 0.0, 40)])
def test_short_sequences_that_the_host_knows_of(nat, keys, gate, cap, more):
    _case(nat, [(keys - 2, 2), (0, min(keys, 33)), (0, 1)] + [(1, 3)] * more, H=8, G=4, d=128, dv=128, page=64, mask=30, keep=2, gate=gate, cap=cap,
          known=True, seed=keys)


@pytest.mark.parametrize("H,G", [(2, 2), (4, 2), (6, 2), (16, 1)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [1, 70, 128, 500, 1024])
def test_sigmoid_weights(nat, H, G, d, window):
    _sigmoid_case(nat, [(0, 63), (3, 64), (0, 65), (500, 130), (8, 2), (11, 1), (900, 300)], H, G, d, window, page=48 if d == 64 else 64)


def test_sigmoid_weights_of_several_items_for_every_cta(nat):
    _sigmoid_case(nat, [(0, 2000), (100, 1500)], 16, 8, 128, 300, page=256)


def test_sigmoid_weights_with_a_negative_scale(nat):
    _sigmoid_case(nat, [(0, 300)], 4, 2, 64, 90, page=16, scale=-0.2)


@pytest.mark.parametrize("H,G", [(16, 8), (4, 4), (8, 1), (6, 2)])
@pytest.mark.parametrize("lens", [(128,), (1, 300, 2, 129, 1), (257, 64, 127), (1000, 700), (2049, 127, 2560, 1, 1800, 600), (300, 129, 1, 256, 40) * 12])
def test_prompts_that_are_their_own_keys(nat, H, G, lens):
    """Strided rows of a packed projection, causal; sequences of one token among them.  Few and short prompts stay with the kernel of one tile a CTA."""
    d, n = 128, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(n + H)
    ud = torch.randn(n, (H + 2 * G) * d + 64, generator=g, device=DEV).to(BF)
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    q, k, v = ud[:, :H * d], ud[:, H * d:(H + G) * d], ud[:, (H + G) * d:(H + 2 * G) * d]
    heads = lambda t, m: t.unflatten(1, (m, d))
    with _Takes(nat, n > 5000):
        out = nat.varlen_attn_prefill(heads(q, H), heads(k, G), heads(v, G), cu, cu, max(lens), max(lens), d ** -0.5)
    ref, o = [], 0
    for m in lens:
        x = ud[o:o + m].to(F64)
        qq, kk, vv = x[:, :H * d].view(m, H, d), x[:, H * d:(H + G) * d].view(m, G, d), x[:, (H + G) * d:(H + 2 * G) * d].view(m, G, d)
        s = torch.einsum("ihd,jhd->hij", qq, kk.repeat_interleave(H // G, 1)) * d ** -0.5
        s = s.masked_fill(torch.ones(m, m, device=DEV).tril() == 0, -math.inf).softmax(-1)
        ref.append(torch.einsum("hij,jhd->ihd", s, vv.repeat_interleave(H // G, 1)))
        o += m
    ref = torch.cat(ref).reshape(n, -1)
    err = (out.reshape(n, -1).to(F64) - ref).abs().max() / ref.abs().max()
    # weights rounded once to 2^-9 and averaged, results rounded to 2^-9
    assert err.item() < 6e-3, err.item()


@pytest.mark.parametrize("lens_q,lens_k", [((300, 130), (300, 130)), ((300, 64, 130), (1000, 64, 131)), ((200, 500, 40, 130), (300, 100, 0, 20))])
def test_prompts_with_key_starts_of_their_own(nat, lens_q, lens_k):
    """Queries are the last of their sequence's tokens; those that would lie in front of its first key see nothing and get zeros."""
    H, G, d = 4, 2, 128
    g = torch.Generator(device=DEV).manual_seed(sum(lens_k))
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(BF)
    cu = lambda lens: torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    q, k, v = r(sum(lens_q), H, d), r(sum(lens_k), G, d), r(sum(lens_k), G, d)
    with _Takes(nat, False):
        out = nat.varlen_attn_prefill(q, k, v, cu(lens_q), cu(lens_k), max(lens_q), max(lens_k), d ** -0.5).view(-1, H, d).to(F64)
    a = b = 0
    for n, m in zip(lens_q, lens_k):
        kk, vv = (t[b:b + m].to(F64).repeat_interleave(H // G, 1) for t in (k, v))
        s = torch.einsum("ihd,jhd->hij", q[a:a + n].to(F64), kk) * d ** -0.5
        seen = torch.arange(m, device=DEV)[None] <= torch.arange(m - n, m, device=DEV)[:, None]
        ref = torch.einsum("hij,jhd->ihd", s.masked_fill(~seen, -math.inf).softmax(-1).nan_to_num(0.0), vv)
        # weights rounded once to 2^-9 and averaged, results rounded to 2^-9
        assert ((out[a:a + n] - ref).abs().max() <= 6e-3 * ref.abs().max()), (n, m)
        a, b = a + n, b + m


@pytest.mark.parametrize("sharp", [0.3, 1, 3, 10])
def test_prompts_are_no_further_from_64_bits_than_tile_by_tile(nat, sharp):
    """Weights rounded once: as far from 64 bits as the kernel for starts of their own, whose largest weight of a row is exact.  (A maximum behind
    the true one leaves that weight a rounding, and a sum of weights before rounding does not take it back: 1.2 times as far.)"""
    n, H, G, d = 2000, 16, 8, 128
    g = torch.Generator(device=DEV).manual_seed(int(sharp * 10))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    q, k, v = (r(n, H, d) * sharp).to(BF), r(n, G, d).to(BF), r(n, G, d).to(BF)
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    s = torch.einsum("ihd,jhd->hij", q.to(F64), k.to(F64).repeat_interleave(H // G, 1)) * d ** -0.5
    ref = torch.einsum("hij,jhd->ihd", s.masked_fill(torch.ones(n, n, device=DEV).tril() == 0, -math.inf).softmax(-1), v.to(F64).repeat_interleave(H // G, 1))
    err = []
    for c in (cu, cu.clone()):
        with _Takes(nat, c is cu):
            out = nat.varlen_attn_prefill(q, k, v, cu, c, n, n, d ** -0.5).view(n, H, d).to(F64)
        err.append(((out - ref).norm() / ref.norm()).item())
    assert err[0] < 1.01 * err[1], err


@pytest.mark.parametrize("sharp", [0.3, 1, 4])
@pytest.mark.parametrize("mask,cap", [(0, 0.0), (64, 0.0), (0, 5.0)])
def test_float_outputs_are_no_further_from_64_bits_than_on_the_other_kernel(nat, sharp, mask, cap):
    """Weights in pairs, outputs in float: the same roundings as the kernel for short sequences, so the same error (1 to 3e-6 here); a fifth
    of it is left for sums in another order."""
    from tests.lm_util import Lay
    n, H, G, d, page = 1000, 4, 2, 128, 64
    g = torch.Generator(device=DEV).manual_seed(mask + int(sharp * 10))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    pages = -(-n // page)
    q, kc, vc = (r(n, H * d) * sharp).to(BF), r(pages, page, G * d).to(BF), r(pages, page, G * d).to(BF)
    k, v = (t.view(-1, G, d)[:n].to(F64).repeat_interleave(H // G, 1) for t in (kc, vc))
    s = torch.einsum("ihd,jhd->hij", q.to(F64).view(n, H, d), k) * d ** -0.5
    s = cap * torch.tanh(s / cap) if cap else s
    dist = torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)[None]
    ok = (dist >= 0) & ((dist < mask) if mask else True)
    ref, err = torch.einsum("hij,jhd->ihd", s.masked_fill(~ok, -math.inf).softmax(-1), v).reshape(n, -1), []
    for known in (0, 1):                                             # 1: said to be short, which is the other kernel's
        lay = Lay([(0, n, list(range(pages)))], page, pages)
        lay.max_keys = known
        out = torch.empty(n, H * d, device=DEV)
        with _Takes(nat, known == 0):
            nat.sink_attn(q, kc, vc, out, lay, None, None, H, G, d, d, page, nat.MASK_WINDOW, mask, d ** -0.5, softcap=cap)
        err.append(((out.to(F64) - ref).norm() / ref.norm()).item())
    assert err[0] < 1.2 * err[1], err


def test_element_gates_in_float(nat):
    """A token that sees itself alone: value times gate, also where the gate leaves next to nothing on (an approximate division answers 0 there).  A few
    roundings of 2^-23, and of 2^-149 where results are that small."""
    from tests.lm_util import Lay
    n, H, G, d, page = 200, 4, 2, 64, 16
    g = torch.Generator(device=DEV).manual_seed(1)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(BF)
    pages = -(-n // page)
    q, kc, vc = r(n, H * d), r(pages, page, G * d), r(pages, page, G * d)
    gate, out = torch.linspace(-88.5, 88, n * H * d, device=DEV).to(BF).view(n, H * d), torch.empty(n, H * d, device=DEV)
    with _Takes(nat):
        nat.sink_attn(q, kc, vc, out, Lay([(0, n, list(range(pages)))], page, pages), None, gate, H, G, d, d, page, nat.MASK_WINDOW, 1, d ** -0.5, gate_el=True)
    ref = vc.view(-1, G, d)[:n].repeat_interleave(H // G, 1).reshape(n, -1).to(F64) * torch.sigmoid(gate.to(F64))
    assert bool(((out - ref).abs() <= ref.abs() * 2 ** -20 + 2 ** -146).all())


@pytest.mark.parametrize("keys", [420, 421])
def test_sigmoid_weights_of_sequences_that_the_host_knows_of(nat, keys):
    _sigmoid_case(nat, [(keys - 40, 40), (0, 33)], 4, 2, 64, 90, page=16, known=True)


@pytest.mark.parametrize("new,more", [(32, 17), (33, 17), (32, 18), (33, 18)])
def test_sigmoid_weights_of_many_short_portions(nat, new, more):
    """Of 148 multiprocessors: 18 sequences of 8 key heads, and 19, which leave portions of up to 32 tokens to the other kernel."""
    _sigmoid_case(nat, [(500, new)] + [(9, 5)] * more, 16, 8, 64, 90, page=64, known=True)


def _sigmoid_case(nat, seqs, H, G, d, window, page, scale=None, known=False):
    from tests.lm_util import Lay
    g = torch.Generator().manual_seed(H * d + window)
    need = [-(-(c + n) // page) for c, n in seqs]
    perm = (torch.randperm(sum(need), generator=g) + 1).tolist()
    tabs = [perm[sum(need[:i]):sum(need[:i + 1])] for i in range(len(need))]
    lay = Lay([(c, n, t) for (c, n), t in zip(seqs, tabs)], page, max(need))
    if known:
        lay.max_keys = max(c + n for c, n in seqs)
    r = lambda *s: torch.randn(s, generator=g, dtype=torch.float32)
    kc, vc = (torch.full((sum(need) + 2, page, G * d), math.nan) for _ in range(2))
    scale = scale if scale is not None else d ** -0.5
    q, r1, r2, pb = r(lay.n_tokens, H * d).to(BF), r(H) * 0.3 + 0.5, r(H).abs(), r(H) - 1.0
    ref, o = [], 0
    for (c, n), t in zip(seqs, tabs):
        k, v = r(c + n, G, d).to(BF), r(c + n, G, d).to(BF)
        at = torch.arange(c + n)
        slot = torch.tensor(t)[at // page] * page + at % page
        kc.view(-1, G * d)[slot], vc.view(-1, G * d)[slot] = k.reshape(c + n, -1).float(), v.reshape(c + n, -1).float()
        x = torch.arange(c, c + n)[:, None] - at[None]
        bias = (r1.to(F64)[:, None, None] * torch.log1p(r2.to(F64)[:, None, None] * x.clamp_min(0)) - pb.to(F64)[:, None, None])
        s = torch.einsum("ihd,jhd->hij", q[o:o + n].view(n, H, d).to(F64), k.to(F64).repeat_interleave(H // G, 1)) * scale - bias
        w = torch.sigmoid(s) * ((x >= 0) & (x < window))
        ref.append(torch.einsum("hij,jhd->ihd", w, v.to(F64).repeat_interleave(H // G, 1)).reshape(n, -1))
        o += n
    ref = torch.cat(ref)
    out = torch.empty(lay.n_tokens, H * d, dtype=BF, device=DEV)
    few = known and (lay.max_keys <= 420 or (lay.max_new <= 32 and G * lay.n_seqs > 148))
    with _Takes(nat, not few and H // G <= 8):               # more heads a key head stay with the plain kernel
        nat.window_sigmoid_attn(q.to(DEV), kc.to(BF).to(DEV), vc.to(BF).to(DEV), out, lay, r1.to(DEV), r2.to(DEV), pb.to(DEV), H, G, d, d, page, window, scale)
    # weights carry 16 bits; the results round to 2^-9
    err = (out.double().cpu() - ref).abs().max() / ref.abs().max()
    assert err.item() < 4e-3, err.item()


@pytest.mark.parametrize("known", [0, 1])                             # 1: said to be short, which is the other kernel's
@pytest.mark.parametrize("off", [-math.inf, torch.finfo(torch.float32).min, -1e31])
@pytest.mark.parametrize("kind,mask", [("window", 50), ("chunk", 100)])
def test_sinks_that_are_off(nat, known, off, kind, mask):
    """A sink of the lowest value is no sink, also for rows that see nothing of their tile's first keys (128 tokens a row tile here)."""
    from tests.lm_util import Lay
    n, H, G, d, page = 400, 2, 2, 64, 16
    g = torch.Generator(device=DEV).manual_seed(5)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(BF)
    pages = -(-n // page)
    q, kc, vc, got = r(n, H * d), r(pages, page, G * d), r(pages, page, G * d), []
    for sink in (None, torch.full((H,), off, device=DEV)):
        lay, out = Lay([(0, n, list(range(pages)))], page, pages), torch.empty(n, H * d, device=DEV)
        lay.max_keys = known
        with _Takes(nat, known == 0):
            nat.sink_attn(q, kc, vc, out, lay, sink, None, H, G, d, d, page, nat.MASK_WINDOW if kind == "window" else nat.MASK_CHUNK,
                          mask, d ** -0.5)
        got.append(out)
    assert torch.equal(*got)


@pytest.mark.parametrize("path", ["softmax", "sigmoid"])
def test_a_wait_that_ran_out_is_an_error(nat, path):
    """The next launch refuses once, and so does the check that the engines make; the next call after that runs again."""
    call = {"softmax": lambda: _case(nat, [(0, 70)]), "sigmoid": lambda: _sigmoid_case(nat, [(0, 70)], 4, 2, 64, 90, page=16)}[path]
    before = nat.portion_attn_timeouts()
    for consumer in (call, nat.check_waits):
        assert nat.lib().b2tts_portion_attn_lose_wait(None) == 0
        torch.cuda.synchronize()
        LOST[0] = nat.portion_attn_timeouts()
        with pytest.raises(RuntimeError, match="prompt portions ran out"):
            consumer()
        nat.check_waits()
        call()
    assert nat.portion_attn_timeouts() == before + 2
