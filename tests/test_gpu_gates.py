"""Activations and gates whose results are rounded to bf16, against 64 bits over every argument that leaves something on: the short convolution's
SiLU and both gates of the group norm, in each of its kernels."""
import pytest
import torch

from tests.lm_util import Lay

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64


def _arguments(n, c):
    """bf16 numbers from -95 to 90, small ones among them."""
    x = torch.cat([torch.linspace(-95, 90, n * c - 4096), torch.linspace(-3, 3, 4096)]).to(BF)
    return x[torch.randperm(n * c, generator=torch.Generator().manual_seed(0))].view(n, c).to(DEV)


def _close(got, ref, more):
    """One rounding to bf16 (2^-8 of a number at most; 2^-134 where results are that small) behind arithmetic good to ``more``."""
    return bool(((got.to(F64) - ref).abs() <= ref.abs() * (2 ** -8 + more) + 2 ** -134 + 2 ** -140).all())


@pytest.mark.parametrize("c", [256, 250])                     # in vectors, one number a thread
def test_silu_of_the_convolution(c):
    import nano_qwen3tts_vllm_b200._native as nat
    n = 512
    x, w, out = _arguments(n, c), torch.zeros(c, 4, device=DEV), torch.empty(n, c, dtype=BF, device=DEV)
    w[:, 3] = 1.0
    lay, state = Lay([(0, n, [0])], n, 1), torch.zeros(1, 3, c, dtype=BF, device=DEV)
    nat.short_conv_act(x, 0, c, w, None, state, lay, out, 4, 1)
    v = x.to(F64)
    # the kernel for odd sizes divides by 1 + e^-x, which overflows at -88.7
    seen = v > (-95 if c == 256 else -88.6)
    assert _close(out[seen], (v * torch.sigmoid(v))[seen], 2 ** -20)


@pytest.mark.parametrize("act", ["sigmoid", "silu"])
@pytest.mark.parametrize("groups,c", [(1, 2048), (16, 2048)])                # a CTA a group, a warp a group
def test_gates_of_the_group_norm(groups, c, act):
    import nano_qwen3tts_vllm_b200._native as nat
    n = 128
    x, out = _arguments(n, c), torch.empty(n, c, dtype=BF, device=DEV)
    y = torch.randn(n, c, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    nat.gated_group_norm(y, x, None, groups, nat.GATE_SIGMOID if act == "sigmoid" else nat.GATE_SILU, False, 1e-6, out)
    v, z = x.to(F64), y.to(F64).view(n, groups, -1)
    g = torch.sigmoid(v) * (v if act == "silu" else 1.0)
    # the norm's float sums and products: a few 2^-23
    assert _close(out, (z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-6)).view(n, c) * g, 2 ** -19)
