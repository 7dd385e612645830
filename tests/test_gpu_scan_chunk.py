"""Recurrences of prompt portions in chunks on the tensor cores against the 64-bit recurrence token by token: portions around the
chunk's edges, carried state, one-token and padding rows beside them, decays from none to total, numbers outside the range of the
three-part split."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.fixture(scope="module")
def nat():
    import nano_qwen3tts_vllm_b200._native as n
    n.lib()
    return n


class Lay:
    """[(position of the first token, new tokens, state slot)]; 0 tokens is a padding row of one packed token."""

    def __init__(self, seqs):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        starts, o = [], 0
        for _, n, _ in seqs:
            starts.append(o)
            o += max(n, 1)
        self.seq_start, self.seq_pos0 = i32(starts), i32([s[0] for s in seqs])
        self.seq_len, self.seq_slot = i32([s[1] for s in seqs]), i32([s[2] for s in seqs])
        self.n_tokens, self.n_seqs, self.starts = o, len(seqs), starts


def _ssm_reference(x, B, C, dt, la, D, S):
    """Outputs and state of one sequence, and the same sums over absolute values (what float roundings are relative to)."""
    n, H, P = x.shape
    rep = H // B.shape[1]
    ys, ya, A = [], [], S.abs()
    for t in range(n):
        b, c = B[t].repeat_interleave(rep, 0), C[t].repeat_interleave(rep, 0)
        g = torch.exp(la[t])[:, None, None]
        up = dt[t][:, None, None] * b[:, :, None] * x[t][:, None, :]
        S, A = g * S + up, g * A + up.abs()
        ys.append(torch.einsum("hnp,hn->hp", S, c) + D[:, None] * x[t])
        ya.append(torch.einsum("hnp,hn->hp", A, c.abs()) + (D[:, None] * x[t]).abs())
    return torch.stack(ys), S, torch.stack(ya), A


def _ssm_case(nat, seqs, H, G, P, N, seed=0, a_log=None, big=None):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay = Lay(seqs)
    n = lay.n_tokens
    xbc, dt_in = r(n, H * P + 2 * G * N).to(torch.bfloat16), r(n, H).to(torch.bfloat16)
    if big is not None:
        row, col, value = big
        xbc[row, col] = value
    dt_bias, D = 0.5 * r(H), r(H)
    a_log = 0.5 * r(H) - 0.5 if a_log is None else torch.full((H,), a_log, device=DEV)
    slots = max(s[2] for s in seqs) + 2
    state = r(slots, H, N, P)
    before, out = state.clone(), torch.full((n, H * P), 3.0, device=DEV)
    nat.ssm_scan(xbc, dt_in, dt_bias, a_log, D, state, out, lay, H, G, P, N)
    dt = torch.nn.functional.softplus(dt_in.float() + dt_bias)                 # the scalars as the float kernel in front forms them
    la = (-torch.exp(a_log) * dt).to(F64)
    for (pos0, m, slot), o in zip(seqs, lay.starts):
        if m == 0:
            continue
        e = slice(o, o + m)
        X = xbc[e].to(F64)
        S0 = before[slot].to(F64) if pos0 else torch.zeros(H, N, P, dtype=F64, device=DEV)
        y, S, ya, A = _ssm_reference(X[:, :H * P].view(m, H, P), X[:, H * P:H * P + G * N].view(m, G, N), X[:, H * P + G * N:].view(m, G, N),
                                     dt[e].to(F64), la[e], D.to(F64), S0)
        yield out[e].view(m, H, P).to(F64), state[slot].to(F64), y, S, ya, A
    used = {s[2] for s in seqs if s[1]}
    for slot in range(slots):
        if slot not in used:
            assert torch.equal(state[slot], before[slot])


def _check(got, state, y, S, ya, A, m):
    """Roundings: one per term of the 128-term sums and a few per token behind them (scalars in float: 2 ulp of the decay each)."""
    u = 2.0 ** -24 * (256 + 8 * m)
    assert bool(((got - y).abs() <= u * ya + 1e-30).all()), ((got - y).abs() / ya).max().item()
    assert bool(((state - S).abs() <= u * A + 1e-30).all())


@pytest.mark.parametrize("P,N,H,G", [(64, 128, 2, 1), (128, 64, 4, 2)])
@pytest.mark.parametrize("n", [2, 15, 16, 17, 63, 64, 65, 128, 130, 197])
def test_state_space_portion_lengths(nat, P, N, H, G, n):
    for case in _ssm_case(nat, [(0, n, 1), (9, n, 0)], H, G, P, N, seed=n):
        _check(*case, n)


def test_state_space_portions_beside_single_tokens_and_padding(nat):
    seqs = [(5, 1, 3), (0, 70, 0), (0, 0, 1), (0, 1, 4), (800, 3, 2)]
    for (got, state, y, S, ya, A), (_, m, _) in zip(_ssm_case(nat, seqs, 2, 1, 64, 128, seed=5), [s for s in seqs if s[1]]):
        _check(got, state, y, S, ya, A, m)


@pytest.mark.parametrize("a_log", [-30.0, 3.0, 6.0])            # no decay, a decay to nothing in a few tokens, in one
def test_state_space_extreme_decays(nat, a_log):
    for case in _ssm_case(nat, [(7, 150, 0)], 2, 1, 64, 128, seed=1, a_log=a_log):
        _check(*case, 150)


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30])
def test_state_space_numbers_outside_the_split(nat, value):
    """They reach the outputs that the recurrence carries them to - the head and value column, from their token on - and the rest of
    the chunk, of the heads and of the columns keeps its values."""
    col = 64 + 5                                               # value column 5 of head 1
    for got, state, y, S, ya, A in _ssm_case(nat, [(3, 100, 0)], 2, 1, 64, 128, seed=2, big=(70, col, value)):
        hit = torch.zeros_like(y, dtype=torch.bool)
        hit[70:, 1, 5] = True
        lost = torch.zeros_like(S, dtype=torch.bool)
        lost[1, :, 5] = True
        clean = lambda t, where: t.masked_fill(where, 0.0)
        _check(clean(got, hit), clean(state, lost), clean(y, hit), clean(S, lost), clean(ya, hit), clean(A, lost), 100)
        if value != 1e30:
            assert not torch.isfinite(got[70:, 1, 5]).any() and not torch.isfinite(state[1, :, 5]).any()
        else:
            assert bool(((got - y).abs()[70:, 1, 5] <= 1e-4 * ya[70:, 1, 5]).all())
