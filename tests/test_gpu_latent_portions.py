"""Latent attention of prompt portions over expanded keys and values: the mixer against the same mixer on absorbed queries and against
64 bits, over portions behind cached tokens, windows, sinks, both kinds of gate, with and without a rotated part."""
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


def _mixer(spec, width, seed, sink):
    from nano_qwen3tts_vllm_b200.models.ridevik import LatentAttentionMixer
    torch.set_default_dtype(BF)
    try:
        with torch.device(DEV):
            m = LatentAttentionMixer(width, spec, 1e-5)
    finally:
        torch.set_default_dtype(torch.float32)
    g = torch.Generator(device=DEV).manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device=DEV) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.2) + (1.0 if p.dim() == 1 else 0.0))
    if not sink:
        m.attn.sink = None
    return m


def _layout(seqs, page):
    from nano_qwen3tts_vllm_b200.engine.sequence import Sequence
    from nano_qwen3tts_vllm_b200.engine.step_layout import MixedStepLayout
    need = [-(-(c + n) // page) for c, n in seqs]
    perm, items = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist(), []
    for i, (c, n) in enumerate(seqs):
        s = Sequence([0] * (c + n))
        s.num_cached_tokens, s.block_table, s.state_slot = c, perm[sum(need[:i]):sum(need[:i + 1])], i
        items.append((s, n))
    lay = MixedStepLayout(sum(n for _, n in seqs), len(seqs), max(need), torch.device(DEV))
    lay.fill(items, page)
    return lay, [s.block_table for s, _ in items], sum(need)


def _reference(m, h, cache, seqs, tables, page):
    s = m.spec
    D = lambda t: t.to(F64)
    rms = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + m.eps) * D(w)
    def turn(v, pos):
        if not s.rot.dims:
            return v
        ang = pos.to(F64)[:, None] * D(m.rotary.freq)
        c, sn = (ang.cos() * m.rotary.mult)[:, None], (ang.sin() * m.rotary.mult)[:, None]
        a, b = v[..., 0:s.rot.dims:2], v[..., 1:s.rot.dims:2]
        return torch.cat([torch.stack([a * c - b * sn, b * c + a * sn], -1).flatten(-2), v[..., s.rot.dims:]], -1)
    u = D(h) @ D(m.in_proj.weight).T
    q = rms(u[:, :s.q_rank], m.q_norm) @ D(m.uq.weight).T if s.q_rank else u[:, :m.q_size]
    out, o, flat = [], 0, D(cache).view(-1, cache.shape[-1])
    for (c, n), bt in zip(seqs, tables):
        x, pos = u[o:o + n, m.q_in:m.q_in + s.kv_rank + s.rot_dim], torch.arange(c, c + n, device=DEV)
        slots = torch.tensor([bt[p // page] * page + p % page for p in range(c + n)], device=DEV)
        flat[slots[c:]] = torch.cat([rms(x[:, :s.kv_rank], m.kv_norm), turn(x[:, None, s.kv_rank:], pos)[:, 0]], -1)
        lat, kr = flat[slots, :s.kv_rank], flat[slots, None, s.kv_rank:].expand(-1, s.heads, s.rot_dim)
        k = torch.cat([torch.einsum("tr,hdr->thd", lat, D(m.uk)), kr], -1)
        v = torch.einsum("tr,hdr->thd", lat, D(m.uv))
        qh = q[o:o + n].view(n, s.heads, s.dim + s.rot_dim)
        qh = torch.cat([qh[..., :s.dim], turn(qh[..., s.dim:], pos)], -1)
        j = torch.arange(c + n, device=DEV)[None]
        ok = (j <= pos[:, None]) & ((pos[:, None] - j < s.window) if s.window else True)
        sc = (torch.einsum("ihd,jhd->hij", qh, k) * s.scale).masked_fill(~ok, -float("inf"))
        if m.attn.sink is not None:
            sc = torch.cat([sc, D(m.attn.sink)[:, None, None].expand(-1, n, 1)], -1)
        a = torch.einsum("hij,jhd->ihd", sc.softmax(-1)[..., :c + n], v)
        if s.gate:
            g = torch.sigmoid(u[o:o + n, m.q_in + s.kv_rank + s.rot_dim:])
            a = a * (g[:, :s.heads, None] if s.head_gate else g.view(n, s.heads, s.vdim))
        out.append(a.reshape(n, -1))
        o += n
    return torch.cat(out) @ D(m.o_proj.weight).T


@pytest.mark.parametrize("dim,rot,vdim,rank,q_rank", [(128, 64, 128, 256, 0), (64, 64, 64, 136, 72), (128, 0, 128, 128, 64), (128, 64, 64, 72, 0)])
@pytest.mark.parametrize("window", [0, 50, 200])
@pytest.mark.parametrize("gate", [None, "head", "element"])
def test_portions_over_expanded_keys(nat, monkeypatch, dim, rot, vdim, rank, q_rank, window, gate):
    from nano_qwen3tts_vllm_b200.config import LatentMixerSpec, RotarySpec
    from nano_qwen3tts_vllm_b200.models.ridevik import LatentAttentionMixer
    from nano_qwen3tts_vllm_b200.utils.context import set_context
    seqs, page, width = [(0, 150), (300, 33), (77, 64), (0, 129)], 16, 128
    spec = LatentMixerSpec(3, dim, rot, vdim, rank, q_rank, window, (dim + rot) ** -0.5, RotarySpec(min(rot, 32), 1e4), gate is not None, gate == "head")
    m = _mixer(spec, width, dim + rot + window, sink=window != 50)
    lay, tables, pages = _layout(seqs, page)
    g = torch.Generator(device=DEV).manual_seed(3)
    h = torch.randn(lay.n_tokens, width, generator=g, device=DEV).to(BF)
    start = torch.randn(pages, page, rank + rot, generator=g, device=DEV).to(BF)
    ref = _reference(m, h, start, seqs, tables, page)
    taken, got = [], {}
    plan = LatentAttentionMixer.expanded_rows
    monkeypatch.setattr(LatentAttentionMixer, "expanded_rows", lambda self, *a: taken.append(plan(self, *a)) or taken[-1])
    monkeypatch.setattr(LatentAttentionMixer, "EXPAND_MIN_PAIRS", 0)
    for least in (32, 1 << 30):
        monkeypatch.setattr(LatentAttentionMixer, "EXPAND_MIN_NEW", least)
        cache = start.clone()
        set_context(False, step_layout=lay)
        with torch.inference_mode():
            launches = nat.portion_attn_launches()
            got[least] = m(h, cache).to(F64)
            assert nat.portion_attn_launches() - launches == (least == 32)
    assert taken[0] is not None and taken[1] is None
    err = {k: ((v - ref).norm() / ref.norm()).item() for k, v in got.items()}
    # both forms round their operands to bf16 at as many places (2^-9 each); the expanded one must not be the worse one
    assert err[32] < 1e-2 and err[32] < 1.15 * err[1 << 30], err
    torch.cuda.synchronize()
    nat.check_waits()


def test_small_portions_and_decoded_tokens_stay_absorbed(nat):
    from nano_qwen3tts_vllm_b200.config import LatentMixerSpec, RotarySpec
    spec = LatentMixerSpec(16, 64, 0, 64, 64, 0, 0, 0.1, RotarySpec(0, 1.0), False)
    m = _mixer(spec, 64, 0, True)
    q, cache = torch.zeros(40, 1024, dtype=BF, device=DEV), torch.zeros(2, 64, 64, dtype=BF, device=DEV)
    for seqs, want in (([(0, 800)], True), ([(0, 700)], False), ([(0, 800), (10, 1)], False), ([(5000, 31), (5000, 31)], False), ([(0, 40)], False)):
        lay, _, _ = _layout(seqs, 64)
        assert (m.expanded_rows(q, None, cache, lay) is not None) == want
