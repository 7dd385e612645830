"""How far the delta rule's chunks are from 64 bits: on the mean of inputs of three sizes no further than with the triangular system of a chunk solved row by row in
floats, for keys that point anywhere and for keys that point the same way, where a solution whose rows are rounded each for itself is."""
import pytest
import torch

from tests.test_gpu_scan_chunk import Lay, _delta_reference

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


# What the rows' substitution measured on these inputs (outputs, state), times 1.005 for inputs that other versions of torch would draw.
@pytest.mark.parametrize("D,alike,outputs,state", [(128, 0.0, 1.051e-7, 9.21e-8), (64, 0.0, 0.998e-7, 9.21e-8), (128, 0.5, 1.164e-7, 9.22e-8), (64, 0.5, 1.095e-7, 9.38e-8),
                                                   (128, 3.0, 1.284e-7, 9.62e-8)])
def test_mean_error(D, alike, outputs, state):
    import nano_qwen3tts_vllm_b200._native as nat
    n, H, G, P, far = 512, 8, 4, 64, []
    for seed in range(1, 17):
        for scale in (0.3, 1.0, 3.0):
            g = torch.Generator(device=DEV).manual_seed(seed)
            r = lambda *s: torch.randn(s, generator=g, device=DEV)
            x = torch.nn.functional.silu(r(n, H * P + 2 * G * D)) * scale
            if alike:
                x[:, G * D:2 * G * D] += alike * r(1, G * D)
            x, gates = x.to(torch.bfloat16), r(n, 2 * H).to(torch.bfloat16)
            a_log, bias, lay = 0.5 * r(H) - 0.5, 0.5 * r(H), Lay([(0, n, 0)])
            lay.max_new = n
            st, out = torch.zeros(1, H, D, P, device=DEV), torch.empty(n, H * P, device=DEV)
            nat.delta_rule_scan(x, gates[:, :H], gates[:, H:], a_log, bias, st, out, lay, H, G, D, P)
            beta, X = torch.sigmoid(gates[:, :H].to(F64)), x.to(F64)
            la = -torch.exp(a_log.to(F64)) * torch.nn.functional.softplus(gates[:, H:].float() + bias).to(F64)
            y, S = _delta_reference(X[:, :G * D].view(n, G, D), X[:, G * D:2 * G * D].view(n, G, D), X[:, 2 * G * D:].view(n, H, P), beta, la,
                                    torch.zeros(H, D, P, dtype=F64, device=DEV))
            y = y.reshape(n, -1)
            far.append((((out.double() - y).norm() / y.norm()).item(), ((st[0].double() - S).norm() / S.norm()).item()))
    got = [sum(f[i] for f in far) / len(far) for i in (0, 1)]
    assert got[0] <= 1.005 * outputs and got[1] <= 1.005 * state, got
