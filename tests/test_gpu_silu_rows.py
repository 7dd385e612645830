"""SiLU and SiLU products over all rows' pieces: rows of one piece, rows that no block fits, calls of one turn, of several and of an odd number of pieces a thread, strided
rows, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _silu64(x):
    return x.double() * torch.sigmoid(x.double())


@pytest.mark.parametrize("inter,rows", [(8, 1), (8, 3), (8, 606208), (8, 606209), (8, 1400001), (40, 3), (264, 1), (264, 40000), (2056, 5), (6144, 1), (6144, 3), (6144, 2369),
                                        (6144, 3001), (65536, 50)])
@pytest.mark.parametrize("mode", ["eager", "fused", "alone", "strided"])
def test_against_64_bits(inter, rows, mode):
    import nano_qwen3tts_vllm_b200._native as nat
    gen = torch.Generator(device=DEV).manual_seed(inter + rows)
    wide = 2 * inter + (8 if mode == "strided" else 0)
    gu = (3 * torch.randn(rows, wide, generator=gen, device=DEV)).to(BF)
    g, u = gu[:, wide - 2 * inter:wide - inter], gu[:, wide - inter:]
    out = torch.full((rows, inter), 7.0, dtype=BF, device=DEV)
    if mode == "alone":
        got = nat.silu_and_mul(g, None, out=out)
    else:
        got = nat.silu_and_mul(g, u, out=out, rounding=nat.ROUND_FUSED if mode == "fused" else nat.ROUND_EAGER)
    for a in range(0, rows, 200000):
        s = slice(a, a + 200000)
        want = _silu64(g[s]) * (1.0 if mode == "alone" else u[s].double())
        # bf16 has 8 significant bits, so a rounding moves a value by at most 2^-8 of it: one rounding, or two where the SiLU is rounded first (2 x 2^-8 + 2^-16); the
        # float arithmetic in front is a few units of 2^-24
        tol = (2 ** -8 if mode in ("alone", "fused") else 2 ** -7) + 2 ** -15
        assert bool(((got[s].double() - want).abs() <= tol * want.abs() + 1e-38).all())
