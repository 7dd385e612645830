"""The router at expert counts around what its warps take at a time, for few tokens (one a CTA) and many, in vectors and number by number."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("experts", [1, 8, 9, 16, 17, 24, 25, 32, 33, 40, 48, 49, 65, 128])
@pytest.mark.parametrize("n,cols", [(5, 512), (700, 512), (700, 510)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_expert_counts(experts, n, cols, dtype):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator(device=DEV).manual_seed(experts + n)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    h, w, top = r(n, cols).to(dtype), r(experts, cols) * cols ** -0.5, min(4, experts)
    i32 = lambda *s: torch.empty(*s, dtype=torch.int32, device=DEV)
    idx, wt, off, pair = i32(n, top), torch.empty(n, top, device=DEV), i32(experts + 1), i32(n * top)
    nat.moe_route(h, w, idx, wt, off, pair, top, 1.0)
    s = torch.sigmoid(h.double() @ w.double().T)
    best, at = s.sort(1, descending=True)
    # float sums of 512 products: scores are good to 1e-6, and choices closer than that may go either way
    clear = (best[:, :top] - torch.cat([best, best.new_zeros(n, 1)], 1)[:, 1:top + 1]).amin(1) > 1e-5
    assert clear.float().mean() > 0.9 and torch.equal(idx[clear].long(), at[clear, :top])
    chosen = s.gather(1, idx.long())
    assert ((wt - chosen / (chosen.sum(1, keepdim=True) + 1e-20)).abs() < 1e-5).all()
    count = torch.bincount(idx.flatten().long(), minlength=experts)
    assert torch.equal(off[1:].long() - off[:-1].long(), count) and torch.equal(idx.flatten()[pair.long()].sort().values, idx.flatten()[pair.long()])
