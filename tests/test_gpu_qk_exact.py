"""Head norms and rotation of steps of many and of few tokens against 64 bits, and with the results on top of the inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _inputs(n, H, G, norm, sections):
    g = torch.Generator().manual_seed(n + H)
    q, k, v = (torch.randn(n, h, 128, generator=g).to(DEV, BF) for h in (H, G, G))
    qw, kw = ((1 + 0.1 * torch.randn(128, generator=g)).to(DEV, BF) if norm else None for _ in range(2))
    pos = torch.randint(0, 4400, (3, n) if sections else (n,), generator=g).to(DEV)
    mod = torch.randint(0, 3, (128,), generator=g).to(DEV, torch.int32) if sections else None
    return q, k, v, qw, kw, pos, mod, (1.0 / 1e6 ** (torch.arange(64) / 64)).to(DEV)


FORMS = [(16, 8, True, False), (3, 1, True, True), (5, 2, False, True), (2, 1, False, False)]


@pytest.mark.parametrize("n", [7, 1183, 1184, 1190])
@pytest.mark.parametrize("H,G,norm,sections", FORMS)
@pytest.mark.parametrize("eager", [True, False])
def test_against_64_bits(n, H, G, norm, sections, eager):
    import nano_qwen3tts_vllm_b200._native as nat
    q, k, v, qw, kw, pos, mod, inv = _inputs(n, H, G, norm, sections)
    got = nat.qknorm_rope_kvwrite(q, k, v, qw, kw, 1e-6, pos, inv, modality=mod, attention_scaling=0.75, rounding=nat.ROUND_EAGER if eager else nat.ROUND_FUSED)
    # the angle is a product of floats by contract; everything behind it in 64 bits
    row = torch.arange(n, device=DEV)
    p = pos if not sections else torch.stack([pos[mod[c].long(), row] for c in range(128)], 1)
    ang = (p.float()[:, None] * inv.repeat(2)[None] if not sections else p.float() * inv.repeat(2)[None]).double()
    c, s = (0.75 * ang.cos())[:, None], (0.75 * ang.sin())[:, None]
    for x, w, y in ((q, qw, got[0]), (k, kw, got[1])):
        x = x.double()
        if norm:
            x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double()
        a, b = x[..., :64], x[..., 64:]
        first, second = (a * c[..., :64], -b * s[..., :64]), (b * c[..., 64:], a * s[..., 64:])
        # a rounding to bf16 moves a value by at most 2^-8 of it: the norm rounds twice (eager) or once, cosines and sines once, each product once, their sum once; the
        # float arithmetic between them is a few units of 2^-24 (cosf and sinf two), which the last term covers
        each = ((2 if eager else 1) if norm else 0) + 2
        for (m, o), part in ((first, y.view(n, -1, 128)[..., :64]), (second, y.view(n, -1, 128)[..., 64:])):
            bound = (each + 1) * 2 ** -8 * 1.02 * (m.abs() + o.abs()) + 1e-6
            assert bool(((part.double() - (m + o)).abs() <= bound).all())


@pytest.mark.parametrize("n", [9, 1184, 1189])
@pytest.mark.parametrize("H,G,norm,sections", FORMS)
def test_results_on_top_of_the_inputs(n, H, G, norm, sections):
    """The contract lets q_out and k_out be q and k where the strides match."""
    import nano_qwen3tts_vllm_b200._native as nat
    q, k, v, qw, kw, pos, mod, inv = _inputs(n, H, G, norm, sections)
    slots = torch.randperm(n, device=DEV).to(torch.int32)
    got = []
    for own in (False, True):
        a, b = q.clone(), k.clone()
        kc, vc = (torch.zeros(n, G, 128, dtype=BF, device=DEV) for _ in range(2))
        extra = dict(q_out=a, k_out=b) if own else {}
        got.append(nat.qknorm_rope_kvwrite(a, b, v, qw, kw, 1e-6, pos, inv, modality=mod, slot_mapping=slots, k_cache=kc, v_cache=vc, **extra) + (kc, vc))
    assert all(torch.equal(x.view(-1), y.view(-1)) for x, y in zip(*got))
