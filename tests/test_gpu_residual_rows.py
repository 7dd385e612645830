"""Residual sums and embeddings with their norm over four columns at a time: row lengths at the edges of what a thread keeps, lengths and addresses that the pieces do not
fit (one column at a time), every optional term, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols", [4, 36, 1020, 1024, 1028, 2048, 2052, 4096, 4100, 4098, 5001])
@pytest.mark.parametrize("off", [0, 1])
def test_against_64_bits(cols, dtype, off):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator().manual_seed(cols + off)
    n, top, eps, gain = 5, 3, 1e-5, torch.tensor([1.3])

    def put(t):                                                       # off: from an address that is no multiple of 16 bytes
        buf = torch.empty(t.numel() + off, dtype=t.dtype, device=DEV)
        buf[off:] = t.flatten().to(DEV)
        return buf[off:].view(t.shape)
    x0 = torch.randn(n, cols, generator=g)
    a, b, z = (torch.randn(m, cols, generator=g).to(dtype) for m in (n, n, n * top))
    zw = torch.rand(n, top, generator=g)

    def check(x, h, exact):
        # sums of at most seven floats, then a norm whose root is that of a sum of squares (positive terms): float rounding a few times over, and one rounding to h's type
        assert bool(((x.cpu().double() - exact).abs() <= 8 * 2 ** -24 * (exact.abs() + 4)).all())
        ref = exact / torch.sqrt((exact * exact).mean(1, keepdim=True) + eps) * gain.double()
        tol = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -18
        assert bool(((h.cpu().double() - ref).abs() <= tol * ref.abs() + 1e-5).all())
    for use in [(1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 0)]:
        x, h = put(x0), put(torch.zeros(n, cols, dtype=dtype))
        nat.residual_norm(x, put(a) if use[0] else None, put(b) if use[1] else None, put(z) if use[2] else None, zw.to(DEV) if use[2] else None, 0.5, h,
                          gain.to(DEV), eps, dtype)
        check(x, h, x0.double() + 0.5 * (use[0] * a.double() + use[1] * b.double() + use[2] * (zw.double()[:, :, None] * z.double().view(n, top, cols)).sum(1)))
    tok, pos = torch.tensor([3, 0, 14, 2, 2], dtype=torch.int32), torch.tensor([0, 4, 1, 3, 2], dtype=torch.int32)
    x, h = put(torch.zeros(n, cols)), put(torch.zeros(n, cols, dtype=dtype))
    nat.embed_pos_norm(tok.to(DEV), pos.to(DEV), put(z), put(a), x, h, gain.to(DEV), eps)
    check(x, h, z.double()[tok.long()] + a.double()[pos.long()])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols", [4, 36, 1020, 1024, 1028, 2048, 2052, 4096])
def test_the_same_bits_whichever_way_a_row_is_read(cols, dtype):
    """An address that is no multiple of 16 bytes sends a row to the kernels of one column at a time: sums, squares and roots are those of four at a time."""
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator().manual_seed(cols)
    n, top, eps, gain = 300, 3, 1e-5, torch.tensor([1.3], device=DEV)
    x0, zw = torch.randn(n, cols, generator=g), torch.rand(n, top, generator=g).to(DEV)
    a, b, z = (torch.randn(m, cols, generator=g).to(dtype) for m in (n, n, n * top))
    tok, pos = (torch.randint(0, n, (n,), generator=g, dtype=torch.int32).to(DEV) for _ in range(2))
    got = []
    for off in (0, 1):
        def put(t):
            buf = torch.empty(t.numel() + off, dtype=t.dtype, device=DEV)
            buf[off:] = t.flatten().to(DEV)
            return buf[off:].view(t.shape)
        for use in [(1, 1, 1), (1, 0, 0), (0, 0, 1)]:
            x, h = put(x0), put(torch.zeros(n, cols, dtype=dtype))
            nat.residual_norm(x, put(a) if use[0] else None, put(b) if use[1] else None, put(z) if use[2] else None, zw if use[2] else None, 0.5, h, gain, eps, dtype)
            got.append((off, x, h))
        x, h = put(torch.zeros(n, cols)), put(torch.zeros(n, cols, dtype=dtype))
        nat.embed_pos_norm(tok, pos, put(a), put(b), x, h, gain, eps)
        got.append((off, x, h))
    for (_, x, h), (_, y, k) in zip(got[:4], got[4:]):
        assert torch.equal(x, y) and torch.equal(h, k)
