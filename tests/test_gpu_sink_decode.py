"""One-token rows of sink attention against 64-bit softmax attention: both CTA sizes (few and many row and head groups), every number of lanes
a cached row is split over with 1, 2 and 4 heads per key head (more scores than lanes, as many, fewer), key counts around a step's 4 keys per
lane group, wide values, page sizes with and without a power of two, masks, kept keys, caps and sinks."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64


@pytest.fixture(scope="module")
def nat():
    import nano_qwen3tts_vllm_b200._native as n
    n.lib()
    return n


def _check(nat, cached, dtype, *, rep, G, d, wide, page, mask=0, keep=0, cap=0.0, sink=True, seed=0):
    from tests.lm_util import Lay
    H, dv = rep * G, d * (2 if wide else 1)
    g = torch.Generator().manual_seed(seed)
    need = [c // page + 1 for c in cached]
    perm = (torch.randperm(sum(need), generator=g) + 1).tolist()
    tabs = [perm[sum(need[:i]):sum(need[:i + 1])] for i in range(len(need))]
    lay = Lay([(c, 1, t) for c, t in zip(cached, tabs)], page, max(need))
    gd = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=gd, device=DEV)
    kc, vc = r(sum(need) + 1, page, G * d).to(dtype), r(sum(need) + 1, page, G * dv).to(dtype)
    q, sk = r(len(cached), H * d).to(dtype), r(H)
    ref = torch.empty(len(cached), H, dv, dtype=F64, device=DEV)
    for b, (c, t) in enumerate(zip(cached, tabs)):
        k = kc[torch.tensor(t, device=DEV)].reshape(-1, G, d)[:c + 1].to(F64).repeat_interleave(rep, 1)
        v = vc[torch.tensor(t, device=DEV)].reshape(-1, G, dv)[:c + 1].to(F64).repeat_interleave(rep, 1)
        j = torch.arange(c + 1, device=DEV)
        s = torch.einsum("hd,jhd->hj", q[b].view(H, d).to(F64), k) * d ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        if mask:
            s = s.masked_fill(~((c - j < mask) | (j < keep)), -math.inf)
        s = torch.cat([s, sk.to(F64)[:, None]], 1) if sink else s
        ref[b] = torch.einsum("hj,jhd->hd", s.softmax(-1)[:, :c + 1], v)
    out = torch.empty(len(cached), H * dv, dtype=torch.float32, device=DEV)
    nat.sink_attn(q, kc, vc, out, lay, sk if sink else None, None, H, G, d, dv, page, nat.MASK_WINDOW, mask, d ** -0.5, keep_first=keep, softcap=cap)
    # operands are exact; float sums over d products and up to 700 keys: 2^-24 * (d + 700) at worst, about 2^-24 * sqrt of it as a rule
    assert ((out.to(F64) - ref.view_as(out)).abs().max() / ref.abs().max()).item() < 1e-5


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
@pytest.mark.parametrize("rep", [1, 2, 3, 4])
@pytest.mark.parametrize("many", [False, True])
def test_sizes(nat, dtype, lanes, rep, many):
    d = lanes * (8 if dtype == BF else 4)
    if d > 256:
        pytest.skip("head sizes up to 256")
    lens = [0, 1, 6, 31, 63, 64, 127, 128, 129, 255, 256, 257, 300, 699]
    for wide in ([False, True] if d <= 128 else [False]):
        _check(nat, lens * 12 if many else lens[::3], dtype, rep=rep, G=2 if many else 1, d=d, wide=wide, page=16, seed=lanes + rep)


@pytest.mark.parametrize("page", [1, 3, 12, 16, 256])
@pytest.mark.parametrize("mask,keep,cap,sink", [(0, 0, 5.0, False), (70, 0, 0.0, True), (70, 9, 30.0, True), (1, 4, 0.0, False), (130, 200, 2.0, False)])
def test_masks_pages_and_caps(nat, page, mask, keep, cap, sink):
    for lens in ([0, 5, 200, 333], [0, 5, 200, 333, 70, 129] * 30):
        _check(nat, lens, BF, rep=2, G=2, d=128, wide=False, page=page, mask=mask, keep=keep, cap=cap, sink=sink, seed=page + mask)


@pytest.mark.parametrize("dtype,out_dtype", [(BF, torch.float32), (BF, BF), (torch.float32, torch.float32)])
@pytest.mark.parametrize("rep,wide", [(1, False), (2, False), (4, True)])
def test_padding_rows_are_zeroed_and_empty_sequences_leave_the_others_alone(nat, dtype, out_dtype, rep, wide):
    from tests.lm_util import Lay
    G, d, page = 2, 64, 16
    H, dv = rep * G, d * (2 if wide else 1)
    gd = torch.Generator(device=DEV).manual_seed(rep)
    r = lambda *s: torch.randn(s, generator=gd, device=DEV)
    kc, vc = r(9, page, G * d).to(dtype), r(9, page, G * dv).to(dtype)
    q, sk = r(5, H * d).to(dtype), r(H)

    def run(lay, rows):
        out = torch.full((len(rows), H * dv), math.nan, dtype=out_dtype, device=DEV)
        nat.sink_attn(q[rows].contiguous(), kc, vc, out, lay, sk, None, H, G, d, dv, page, nat.MASK_WINDOW, 0, d ** -0.5)
        return out

    live = {1: (40, 1, [1, 2, 3]), 3: (3, 1, [4])}
    ref = run(Lay([live[1], live[3]], page, 3), [1, 3])
    padded = run(Lay([(0, 0, [0]), live[1], (0, 0, [0]), live[3], (0, 0, [0])], page, 3), [0, 1, 2, 3, 4])
    assert torch.equal(padded[[1, 3]], ref) and (padded[[0, 2, 4]] == 0).all()
    lay = Lay([live[1], live[3]], page, 3)                     # a sequence without tokens and without a row between them
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lay.seq_start, lay.seq_pos0, lay.seq_len, lay.seq_slot = i32([0, 1, 1]), i32([40, 0, 3]), i32([1, 0, 1]), i32([0, 1, 2])
    lay.tok_seq, lay.n_seqs = i32([0, 2]), 3
    lay.block_tables = lay.block_tables[[0, 0, 1]].contiguous()
    assert torch.equal(run(lay, [1, 3]), ref)


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("lens,tok_seq", [([1, 0, 1], [0, 2, 1]), ([0, 1, 1, 0], [1, 2, 0, 3]), ([1, 0, 0, 1], [1, 0, 3, 2])])
def test_padding_rows_lie_where_their_tokens_say(nat, dtype, lens, tok_seq):
    """A row is padding where its own sequence brings no token; where empty sequences start - here a running sum, which names other sequences'
    rows, or a number beyond all rows - means nothing."""
    from tests.lm_util import Lay
    G, d, page, H, n = 2, 64, 16, 4, len(lens)
    gd = torch.Generator(device=DEV).manual_seed(n)
    r = lambda *s: torch.randn(s, generator=gd, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    kc, vc, q, sk = r(9, page, G * d).to(dtype), r(9, page, G * d).to(dtype), r(n, H * d).to(dtype), r(H)
    cached = [40 - 9 * b for b in range(n)]
    lay = Lay([(c, 1, [1 + b, 4 + b, 2]) for b, c in enumerate(cached)], page, 3)
    run = lambda rows, lay: (nat.sink_attn(q[rows].contiguous(), kc, vc, o := torch.full((len(rows), H * d), math.nan, dtype=dtype, device=DEV), lay, sk, None,
                                           H, G, d, d, page, nat.MASK_WINDOW, 0, d ** -0.5), o)[1]
    row_of = {b: t for t, b in enumerate(tok_seq)}
    ref = run([row_of[b] for b in range(n)], lay)                # every sequence with a token, in order
    for starts in ([sum(lens[:b]) for b in range(n)], [1 << 20] * n):
        lay.seq_len, lay.tok_seq = i32(lens), i32(tok_seq)
        lay.seq_start = i32([row_of[b] if m else starts[b] for b, m in enumerate(lens)])
        lay.positions = i32([cached[b] for b in tok_seq])
        out = run(list(range(n)), lay)
        for b, m in enumerate(lens):
            assert torch.equal(out[row_of[b]], ref[b]) if m else bool((out[row_of[b]] == 0).all()), (b, starts)
