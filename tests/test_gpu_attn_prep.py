"""Preparation of attention steps in 16-byte pieces (bf16) against 64 bits: both norms, both pairings, tied values, layers without caches,
padding rows, and token counts around the lines where the kernels change."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64


class _Lay:
    pass


def _turn(x, ang, interleaved):
    """x [n, heads, d], ang [n, rot_dims / 2]."""
    h = ang.shape[1]
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    r = x[..., :2 * h]
    a, b = (r[..., 0::2], r[..., 1::2]) if interleaved else (r[..., :h], r[..., h:])
    y = (a * c - b * s, b * c + a * s)
    r = torch.stack(y, -1).flatten(-2) if interleaved else torch.cat(y, -1)
    return torch.cat([r, x[..., 2 * h:]], -1)


@pytest.mark.parametrize("n", [1, 2, 295, 296, 1183, 1184, 1185])
@pytest.mark.parametrize("head_norm,norm,rot,interleaved,tied,d,dv", [
    (False, False, 0, True, False, 128, 64), (False, False, 64, True, False, 128, 128), (False, True, 32, False, True, 32, 32),
    (True, True, 128, True, False, 128, 128), (True, True, 64, False, False, 64, 40), (True, False, 16, False, False, 256, 256), (True, True, 0, True, False, 32, 8)])
def test_against_64_bits(n, head_norm, norm, rot, interleaved, tied, d, dv):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator().manual_seed(n + d + rot)
    H, G, extra, eps = 6, 2, 8, 1e-5
    nq, nk, nv = H * d, G * d, G * dv
    u = torch.randn(n, extra + nq + nk + nv, generator=g).to(BF)
    qb, kb, vb = (torch.randn(x, generator=g) for x in (nq, nk, nv))
    qw, kw = (torch.rand(d if head_norm else x, generator=g) + 0.5 for x in (nq, nk))
    freq = torch.rand(rot // 2, generator=g)
    lay = _Lay()
    lay.n_tokens, pos = n, torch.randint(0, 300, (n,), generator=g)
    slots = torch.randperm(n + 3, generator=g)[:n]
    if n > 2:
        slots[n // 2] = -1                                            # a padding row
    dev = lambda t, dt=None: t.to(DEV, dt) if dt else t.to(DEV)
    lay.positions, lay.slot_mapping = dev(pos, torch.int32), dev(slots, torch.int32)
    ang = pos.float()[:, None] * freq                                 # as the kernels form it
    x = u.to(F64)
    q, k = x[:, extra:extra + nq] + qb, x[:, extra + nq:extra + nq + nk] + kb
    v = k if tied else x[:, extra + nq + nk:] + vb
    q, k = q.view(n, H, d), k.view(n, G, d)
    if norm:
        rms = lambda t, w: (t / torch.sqrt((t * t).mean(-1, keepdim=True) + eps) * w)
        q, k = (rms(q, qw), rms(k, kw)) if head_norm else (rms(q.flatten(1), qw).view(n, H, d), rms(k.flatten(1), kw).view(n, G, d))
    q, k = _turn(q, ang.to(F64), interleaved), _turn(k, ang.to(F64), interleaved)
    qo = torch.full((n, nq), 7.0, dtype=BF, device=DEV)
    kc, vc = torch.full((n + 3, 1, nk), 7.0, dtype=BF, device=DEV), torch.full((n + 3, 1, nv), 7.0, dtype=BF, device=DEV)
    args = [dev(u), extra, extra + nq, -1 if tied else extra + nq + nk, dev(qb), dev(kb), dev(vb), dev(qw) if norm else None, dev(kw) if norm else None]
    if head_norm:
        table = torch.cat([ang.cos(), ang.sin()], 1).contiguous()
        nat.attn_head_prep(*args, dev(table) if rot else None, interleaved, lay, qo, kc, vc, H, G, d, dv, eps)
    else:
        nat.attn_prep(*args, dev(freq) if rot else None, rot, lay, qo, kc, vc, H, G, d, dv, eps, interleaved=interleaved)
    live = slots >= 0
    # one rounding to bf16 (2^-9 of the number) behind float arithmetic on numbers of this size
    close = lambda a, b: bool(((a.double().cpu() - b).abs() <= b.abs() * 2 ** -8 * 1.01 + 1e-4).all())
    assert close(qo[live.to(DEV)], q.flatten(1)[live]) and bool((qo[~live.to(DEV)] == 7).all())
    at = slots[live].to(DEV)
    assert close(kc[at, 0], k.flatten(1)[live]) and close(vc[at, 0], v.flatten(1)[live])
    other = torch.ones(n + 3, dtype=torch.bool, device=DEV)
    other[at] = False
    assert bool((kc[other] == 7).all()) and bool((vc[other] == 7).all())
    if not head_norm and not tied:
        q2 = torch.empty_like(qo)
        nat.attn_prep(args[0], extra, 0, 0, args[4], None, None, args[7], torch.ones(nk, device=DEV) if norm else None, dev(freq) if rot else None,
                      rot, lay, q2, None, None, H, G, d, dv, eps, interleaved=interleaved)
        assert torch.equal(q2[live.to(DEV)], qo[live.to(DEV)])
