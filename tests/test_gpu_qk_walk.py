"""Head norms and rotation of many tokens, each thread with its piece of a head over a run of tokens: the same bits as steps of few tokens give, for every remainder
of a run, with and without norms, sectioned positions, caches and padding rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


@pytest.mark.parametrize("n", list(range(1184, 1192)))
@pytest.mark.parametrize("H,G,norm,sections,cache,eager", [(16, 8, True, False, True, True), (3, 1, True, True, True, False), (5, 2, False, True, False, True),
                                                           (2, 1, False, False, True, True)])
def test_same_bits_as_few_tokens(n, H, G, norm, sections, cache, eager):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator().manual_seed(n + H)
    u = torch.randn(n, (H + 2 * G) * 128 + 8, generator=g).to(DEV, BF)[:, 8:]
    q, k, v = (t.unflatten(1, (-1, 128)) for t in u.split([H * 128, G * 128, G * 128], 1))
    qw, kw = ((1 + 0.1 * torch.randn(128, generator=g)).to(DEV, BF) if norm else None for _ in range(2))
    pos = torch.randint(0, 4400, (3, n) if sections else (n,), generator=g).to(DEV)
    mod = torch.randint(0, 3, (128,), generator=g).to(DEV, torch.int32) if sections else None
    inv = (1.0 / 1e6 ** (torch.arange(64) / 64)).to(DEV)
    slots = torch.randperm(n, generator=g).to(DEV, torch.int32)
    slots[n // 2] = -1

    def run(cuts):
        kc, vc = (torch.full((n, G, 128), 7.0, dtype=BF, device=DEV) for _ in range(2))
        out = []
        for a, b in zip(cuts, cuts[1:]):
            extra = dict(slot_mapping=slots[a:b].contiguous(), k_cache=kc, v_cache=vc) if cache else {}
            out.append(nat.qknorm_rope_kvwrite(q[a:b], k[a:b], v[a:b] if cache else None, qw, kw, 1e-6, pos[..., a:b].contiguous(), inv, modality=mod,
                                               rounding=nat.ROUND_EAGER if eager else nat.ROUND_FUSED, **extra))
        return [torch.cat([o[i] for o in out]) for i in range(2)] + [kc, vc]
    for a, b in zip(run([0, n]), run([0, 600, n])):
        assert torch.equal(a, b)
