"""The streaming row kernels at the edges of their runs and vectors: the causal convolution against a 64-bit one (runs of eight tokens, carried rows,
filters off a 16-byte boundary), the gated group norm around the vectors a thread keeps, the squared ReLU around its vectors."""
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


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("channels", [8, 264, 1040])
def test_convolution_runs(nat, dtype, taps, off, channels):
    from tests.lm_util import Lay
    seqs = [(0, 1), (0, 7), (1, 8), (2, 9), (40, 17), (0, 33)]
    lay = Lay([(c, n, [i + 1]) for i, (c, n) in enumerate(seqs)], 64, 1)
    g = torch.Generator(device=DEV).manual_seed(taps)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    u, w, bias = r(lay.n_tokens, channels + 16).to(dtype), r(channels * taps + off)[off:].view(channels, taps), r(channels)
    state, out = r(len(seqs) + 8, taps - 1, channels).to(dtype), torch.empty(lay.n_tokens, channels, dtype=dtype, device=DEV)
    before, slots, o = state.clone(), lay.seq_slot.tolist(), 0
    nat.short_conv_act(u, 8, channels, w, bias, state, lay, out, taps)
    for (c, n), slot in zip(seqs, slots):
        rows = torch.cat([before[slot], u[o:o + n, 8:8 + channels]]).to(F64)
        if c < taps - 1:
            rows[:taps - 1 - c] = 0
        ref = bias.to(F64) + sum(w[:, j].to(F64) * rows[j:j + n] for j in range(taps))
        ref = ref * torch.sigmoid(ref)
        # float sums of up to five terms below 16; bf16 results round to 2^-9 of themselves
        assert ((out[o:o + n].to(F64) - ref).abs() <= 1e-5 + ref.abs() * (2 ** -8 if dtype == BF else 1e-5)).all()
        assert torch.equal(state[slot].to(F64), rows[n:])
        o += n


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("cols,groups", [(4, 1), (1020, 1), (1024, 1), (4096, 1), (4100, 1), (4096, 2), (2048, 16), (1536, 3), (520, 130)])
@pytest.mark.parametrize("act,first,gate", [(0, False, True), (1, True, True), (1, False, False)])
def test_gated_group_norm(nat, dtype, cols, groups, act, first, gate):
    g = torch.Generator(device=DEV).manual_seed(cols + groups)
    y, z = torch.randn(5, cols, generator=g, device=DEV), torch.randn(5, cols + 8, generator=g, device=DEV).to(dtype)
    w, out = torch.randn(cols, generator=g, device=DEV), torch.empty(5, cols, dtype=dtype, device=DEV)
    nat.gated_group_norm(y, z[:, 8:] if gate else None, w, groups, act, first, 1e-5, out)
    zz = z[:, 8:].to(F64)
    gg = (torch.sigmoid(zz) * (zz if act else 1.0)) if gate else torch.ones_like(zz)
    v = (y.to(F64) * (gg if first else 1.0)).view(5, groups, -1)
    ref = (v * (v.square().mean(-1, keepdim=True) + 1e-5).rsqrt()).view(5, cols) * w.to(F64) * (1.0 if first else gg)
    assert ((out.to(F64) - ref).abs() <= 1e-5 + ref.abs() * (2 ** -8 if dtype == BF else 1e-5)).all()


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("n", [1, 4, 7, 8, 2047, 2048, 2056, 8192, 8200, 100008])
@pytest.mark.parametrize("off", [0, 1])
def test_squared_relu(nat, dtype, n, off):
    y = torch.randn(n + off + 8, device=DEV).to(dtype)
    ref = y.clone()
    ref[off:off + n] = y[off:off + n].float().clamp_min(0).square().to(dtype)
    nat.relu_sq_(y[off:off + n])
    assert torch.equal(y, ref)
