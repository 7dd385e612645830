"""SiLU and SiLU products over all rows' pieces: rows of one piece, rows that no block fits, calls of one turn, of several and of an odd number of pieces a thread, strided
rows, against 64 bits; and every gate that bf16 has."""
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


def test_every_gate():
    """All bf16 values: the quotient g / (1 + e^-g) of floats, rounded once, as the epilogues of the products form it."""
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.arange(65536, dtype=torch.int32, device=DEV).to(torch.int16).view(BF).view(512, 128)
    one, up = torch.ones_like(g), torch.full_like(g, 1.2421875)
    f = g.float() / (1 + torch.exp(-g.float()))
    same = lambda x, y: torch.equal(x.isnan(), y.isnan()) and torch.equal(x[~x.isnan()], y[~y.isnan()])
    assert same(nat.silu_and_mul(g, None), f.to(BF))
    assert same(nat.silu_and_mul(g, one), f.to(BF))
    assert same(nat.silu_and_mul(g, up), f.to(BF) * up)
    assert same(nat.silu_and_mul(g, up, rounding=nat.ROUND_FUSED), (f * up.float()).to(BF))


def test_fused_products_of_every_gate():
    """With fused rounding the SiLU meets the other factor as a float: factors that leave the rounding of the product to its last bits."""
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.arange(65536, dtype=torch.int32, device=DEV).to(torch.int16).view(BF).view(512, 128)
    f = g.float() / (1 + torch.exp(-g.float()))
    for up in (1.0078125, 1.109375, 0.703125, 1.9921875, 3.015625e-3):
        u = torch.full_like(g, up)
        got, want = nat.silu_and_mul(g, u, rounding=nat.ROUND_FUSED), (f * u.float()).to(BF)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~got.isnan()], want[~want.isnan()])
