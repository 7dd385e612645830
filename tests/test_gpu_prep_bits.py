"""Attention steps of many tokens (a thread walks its piece of the row) give each token the bits that it has in a step of fewer tokens (a CTA a token)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF = "cuda:0", torch.bfloat16


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("d,rot", [(32, 16), (64, 64), (128, 32), (128, 128), (256, 256)])
def test_a_token_has_the_same_bits_among_many_and_few(d, rot, interleaved, norm):
    import nano_qwen3tts_vllm_b200._native as nat
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    H, G, few, n = 6, 2, 3 * sms, 32 * sms + 5
    g = torch.Generator(device=DEV).manual_seed(d + rot + 2 * interleaved + norm)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    u, qb, kb, vb = rnd(n, (H + 2 * G) * d).to(BF), rnd(H * d), rnd(G * d), rnd(G * d)
    qw, kw = (rnd(d) * 0.1 + 1, rnd(d) * 0.1 + 1) if norm else (None, None)
    ang = 300 * rnd(n, rot // 2)
    table = torch.cat([ang.cos(), ang.sin()], 1).contiguous()

    def step(lo, hi):
        m = hi - lo
        at = torch.arange(m, dtype=torch.int32, device=DEV)
        lay = types.SimpleNamespace(n_tokens=m, positions=at, slot_mapping=at)
        q, k, v = (torch.zeros(m, x * d, dtype=BF, device=DEV) for x in (H, G, G))
        nat.attn_head_prep(u[lo:hi], 0, H * d, (H + G) * d, qb, kb, vb, qw, kw, table[lo:hi], interleaved, lay, q, k.view(m, 1, -1), v.view(m, 1, -1),
                           H, G, d, d, 1e-6)
        return q, k, v

    many = step(0, n)
    for lo in [*range(0, n - few, few), n - few]:
        for name, a, b in zip("qkv", many, step(lo, lo + few)):
            assert torch.equal(a[lo:lo + few].view(torch.int16), b.view(torch.int16)), (name, lo)
