"""Recurrences of prompt portions in chunks on the tensor cores against the 64-bit recurrence token by token: portions around the
chunk's edges, carried state, one-token and padding rows beside them, decays from none to total, numbers outside the range of the
three-part split."""
import math

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


def _strong_gates(x, a_log, rows):
    """Gate pre-activations whose decays are e^-1 or so, but for a token in 23 with about e^(-0.7 e^a_log)."""
    x = 0.5 * x - a_log
    x[5 % rows::23] = 0.0
    return x


def _ssm_case(nat, seqs, H, G, P, N, seed=0, a_log=None, big=None, strong=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay = Lay(seqs)
    n = lay.n_tokens
    xbc, dt_in = r(n, H * P + 2 * G * N).to(torch.bfloat16), r(n, H).to(torch.bfloat16)
    if strong:
        dt_in = _strong_gates(dt_in.float(), a_log, n).to(torch.bfloat16)
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


@pytest.mark.parametrize("magnitude", [1e6, 1e9, 1e12, 1e16, 1e20, 1e30])
def test_state_space_gates_far_beyond_a_total_decay(nat, magnitude):
    """The token forgets everything; what the tokens behind it forget is as little as ever."""
    for case in _ssm_case(nat, [(7, 150, 0)], 2, 1, 64, 128, seed=3, a_log=math.log(magnitude), strong=True):
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


# ------------------------------------------------------------------------------------------------ delta rule
def _delta_reference(q, k, v, beta, la, S):
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    n, H, P = v.shape
    rep = H // q.shape[1]
    q, k = unit(q) * q.shape[-1] ** -0.5, unit(k)
    ys = []
    for t in range(n):
        kt, qt = k[t].repeat_interleave(rep, 0), q[t].repeat_interleave(rep, 0)
        S = torch.exp(la[t])[:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hdp,hd->hp", S, kt))
        S = S + kt[:, :, None] * u[:, None, :]
        ys.append(torch.einsum("hdp,hd->hp", S, qt))
    return torch.stack(ys), S


def _delta_case(nat, seqs, H, G, D, P, seed=0, a_log=None, alike=0.0, big=None, strong=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay = Lay(seqs)
    n = lay.n_tokens
    qkv = r(n, 2 * G * D + H * P)
    qkv[:, G * D:2 * G * D] += alike * r(1, G * D)             # keys that point the same way: the solve's off-diagonal is dense
    qkv, ba = qkv.to(torch.bfloat16), r(n, 2 * H).to(torch.bfloat16)
    if strong:
        ba[:, H:] = _strong_gates(ba[:, H:].float(), a_log, n).to(torch.bfloat16)
    if big is not None:
        row, col, value = big
        qkv[row, col] = value
    a_log = 0.5 * r(H) - 0.5 if a_log is None else torch.full((H,), a_log, device=DEV)
    dt_bias = 0.5 * r(H)
    slots = max(s[2] for s in seqs) + 2
    state = r(slots, H, D, P)
    before, out = state.clone(), torch.full((n, H * P), 3.0, device=DEV)
    nat.delta_rule_scan(qkv, ba[:, :H], ba[:, H:], a_log, dt_bias, state, out, lay, H, G, D, P)
    beta = torch.sigmoid(ba[:, :H].to(F64))
    la = -torch.exp(a_log.to(F64)) * torch.nn.functional.softplus(ba[:, H:].float() + dt_bias).to(F64)
    for (pos0, m, slot), o in zip(seqs, lay.starts):
        if m == 0:
            continue
        e = slice(o, o + m)
        X = qkv[e].to(F64)
        S0 = before[slot].to(F64) if pos0 else torch.zeros(H, D, P, dtype=F64, device=DEV)
        y, S = _delta_reference(X[:, :G * D].view(m, G, D), X[:, G * D:2 * G * D].view(m, G, D), X[:, 2 * G * D:].view(m, H, P), beta[e], la[e], S0)
        yield out[e].view(m, H, P).to(F64), state[slot].to(F64), y, S
    used = {s[2] for s in seqs if s[1]}
    for slot in range(slots):
        if slot not in used:
            assert torch.equal(state[slot], before[slot])


def _check_delta(got, state, y, S, m):
    """A write moves the state by a contraction, so roundings add up: a few hundred per token's sums at first (128 terms, three of
    them), a few per token afterwards, relative to the largest numbers of the state; an output adds 128 of them, scaled by 128^-0.5."""
    u = 2.0 ** -24 * (512 + 8 * m) * max(S.abs().max().item(), 1.0)
    assert (got - y).abs().max().item() <= u and (state - S).abs().max().item() <= u, ((got - y).abs().max().item(), (state - S).abs().max().item(), u)


@pytest.mark.parametrize("D,P,H,G", [(128, 64, 2, 1), (64, 128, 4, 2)])
@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 63, 64, 65, 128, 131, 200])
def test_delta_rule_portion_lengths(nat, D, P, H, G, n):
    for case in _delta_case(nat, [(0, n, 1), (9, n, 0)], H, G, D, P, seed=n):
        _check_delta(*case, n)


def test_delta_rule_portions_beside_single_tokens_and_padding(nat):
    seqs = [(5, 1, 3), (0, 70, 0), (0, 0, 1), (0, 1, 4), (800, 3, 2)]
    for case, (_, m, _) in zip(_delta_case(nat, seqs, 2, 2, 128, 128, seed=5), [s for s in seqs if s[1]]):
        _check_delta(*case, m)


@pytest.mark.parametrize("a_log,alike", [(-30.0, 0.0), (6.0, 0.0), (-30.0, 4.0), (-30.0, 100.0)])
def test_delta_rule_extreme_decays_and_keys_that_point_the_same_way(nat, a_log, alike):
    for case in _delta_case(nat, [(7, 150, 0)], 2, 1, 128, 64, seed=1, a_log=a_log, alike=alike):
        _check_delta(*case, 150)


@pytest.mark.parametrize("magnitude", [1e6, 1e9, 1e12, 1e16, 1e20, 1e30])
def test_delta_rule_gates_far_beyond_a_total_decay(nat, magnitude):
    for case in _delta_case(nat, [(7, 150, 0)], 2, 1, 128, 64, seed=3, a_log=math.log(magnitude), strong=True):
        _check_delta(*case, 150)


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30])
def test_delta_rule_values_outside_the_split(nat, value):
    """A value's column of its head is lost from its token on; everything else keeps its numbers."""
    col = 2 * 128 + 64 + 5                                     # value column 5 of head 1
    for got, state, y, S in _delta_case(nat, [(3, 100, 0)], 2, 1, 128, 64, seed=2, big=(70, col, value)):
        hit, lost = torch.zeros_like(y, dtype=torch.bool), torch.zeros_like(S, dtype=torch.bool)
        hit[70:, 1, 5] = lost[1, :, 5] = True
        _check_delta(got.masked_fill(hit, 0.0), state.masked_fill(lost, 0.0), y.masked_fill(hit, 0.0), S.masked_fill(lost, 0.0), 100)
        if value != 1e30:
            assert not torch.isfinite(got[70:, 1, 5]).any()
        else:
            assert bool(((got - y)[70:, 1, 5].abs() <= 1e-4 * y[70:, 1, 5].abs().max()).all())


# ------------------------------------------------------------------------------------------------ beside the token-by-token kernel
def _inputs(kind, tokens, seed, scale=1.0, D=128, P=64):
    """[sequences x tokens] inputs of 8 heads as a model has them, and what runs rows of them (as they are packed) on states."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    H, G, silu = 8, (1 if kind == "ssm" else 4), torch.nn.functional.silu
    x = (silu(r(*tokens, (H * P + 2 * G * D))) * scale).to(torch.bfloat16)
    gates = r(*tokens, H if kind == "ssm" else 2 * H).to(torch.bfloat16)
    a_log, bias, skip = 0.5 * r(H) - 0.5, 0.5 * r(H), 0.5 * r(H)

    def run(nat, seqs, rows_x, rows_g, state, max_new=0):
        lay = Lay(seqs)
        lay.max_new = max_new
        out = torch.empty(lay.n_tokens, H * P, device=DEV)
        if kind == "ssm":
            nat.ssm_scan(rows_x, rows_g, bias, a_log, skip, state, out, lay, H, G, P, D)
        else:
            nat.delta_rule_scan(rows_x, rows_g[:, :H], rows_g[:, H:], a_log, bias, state, out, lay, H, G, D, P)
        return out
    return x, gates, (a_log, bias, skip), run, H, G


@pytest.mark.parametrize("kind", ["ssm", "delta"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scalars_of_one_token_steps_are_float(nat, kind, dtype):
    """The step of a decoding sequence forms its decay with float functions, whatever runs beside it: with nothing written (keys and values
    zero) the state is the old one times that decay, bit for bit."""
    x, gates, (a_log, bias, skip), run, H, G = _inputs(kind, (64, 1), 4)
    gates = gates[:, 0].to(dtype).contiguous()
    state = torch.randn(64, H, 128, 64, device=DEV)
    z = gates[:, -H:].float() + bias
    decay = torch.exp(-(torch.exp(a_log) * (z.clamp(min=0) + torch.log1p(torch.exp(-z.abs())))))
    want = state * decay[:, :, None, None]
    run(nat, [(9, 1, i) for i in range(64)], torch.zeros_like(x[:, 0]).to(dtype), gates, state)
    assert torch.equal(state, want)


@pytest.mark.parametrize("kind", ["ssm", "delta"])
def test_short_portions_are_walked_token_by_token(nat, kind):
    """A portion of a few tokens gives the bits of as many one-token steps, alone, beside others and beside a portion that runs in chunks."""
    x, gates, _, run, H, G = _inputs(kind, (6, 300), 1)
    for n in (2, 6, 12):
        long = 300
        state = torch.zeros(7, H, 128, 64, device=DEV)
        steps = torch.stack([run(nat, [(t, 1, i) for i in range(5)], x[:5, t].contiguous(), gates[:5, t].contiguous(), state) for t in range(n)], 1)
        for seqs in ([(0, n, i) for i in range(5)], [(0, n, i) for i in range(5)] + [(0, long, 5)]):
            rows = lambda v: torch.cat([v[i, :m] for i, (_, m, _) in enumerate(seqs)])
            whole = torch.zeros_like(state)
            out = run(nat, seqs, rows(x), rows(gates), whole)
            assert torch.equal(out[:5 * n].view(5, n, -1), steps) and torch.equal(whole[:5], state[:5])


@pytest.mark.parametrize("kind", ["ssm", "delta"])
def test_the_longest_portion_may_be_given_too_long(nat, kind):
    """``max_new`` is a bound: portions below it, alone or beside others, come out the same (float roundings apart)."""
    x, gates, _, run, H, G = _inputs(kind, (3, 70), 5)
    for lens in ([1], [5], [70], [5, 1], [70, 5, 1]):
        seqs = [(0, m, i) for i, m in enumerate(lens)]
        rows = lambda v: torch.cat([v[i, :m] for i, m in enumerate(lens)])
        outs, states = [], []
        for max_new in (0, max(lens), 200):
            states.append(torch.zeros(4, H, 128, 64, device=DEV))
            outs.append(run(nat, seqs, rows(x), rows(gates), states[-1], max_new))
        for o, S in zip(outs[1:], states[1:]):
            assert (o - outs[0]).norm() <= 1e-6 * outs[0].norm() and (S - states[0]).norm() <= 1e-6 * states[0].norm()


@pytest.mark.parametrize("D,P", [(128, 64), (64, 128)])
@pytest.mark.parametrize("n", [25, 33, 41, 49, 79, 80, 81, 95, 112, 127])
def test_last_chunks_of_every_number_of_blocks(nat, n, D, P):
    """Portions just above what is walked, and last chunks on either side of each block of 16 tokens."""
    for case in _ssm_case(nat, [(0, n, 1), (9, n, 0)], 2, 1, P, D, seed=n):
        _check(*case, n)
    for case in _delta_case(nat, [(0, n, 1), (9, n, 0)], 2, 1, D, P, seed=n):
        _check_delta(*case, n)


@pytest.mark.parametrize("kind", ["ssm", "delta"])
@pytest.mark.parametrize("D,P", [(128, 64), (64, 64)])
def test_no_precision_is_given_up_in_chunks(nat, kind, D, P):
    """The norms of the errors against 64 bits over 512 tokens, outputs and state, are on average over eight inputs of three sizes not above
    the token-by-token kernel's (the same inputs in portions of 10), which are about 1e-7.  Without the third part of a split it is 1.4 times
    that (state against queries and keys) to 2e-6 (weights, update)."""
    B, n, totals = 2, 512, torch.zeros(4, dtype=F64)
    for seed in range(1, 9):
        x, gates, (a_log, bias, skip), run, H, G = _inputs(kind, (B, n), seed, (1.0, 0.3, 3.0)[seed % 3], D, P)
        state = torch.zeros(B, H, D, P, device=DEV)
        out = run(nat, [(0, n, i) for i in range(B)], x.view(B * n, -1), gates.view(B * n, -1), state).view(B, n, H, P)
        walked_state, walked = torch.zeros_like(state), []
        for t in range(0, n, 10):
            m = min(10, n - t)
            walked.append(run(nat, [(t, m, i) for i in range(B)], x[:, t:t + m].reshape(B * m, -1), gates[:, t:t + m].reshape(B * m, -1),
                              walked_state).view(B, m, H, P))
        # both sequences at once, as heads of one
        X, u = x.to(F64).transpose(0, 1), gates.to(F64).transpose(0, 1)
        heads = lambda t, h: t.reshape(n, B * h, -1)
        S0 = torch.zeros(B * H, D, P, dtype=F64, device=DEV)
        if kind == "ssm":
            dt = torch.nn.functional.softplus(u + bias.to(F64))
            y, S, _, _ = _ssm_reference(heads(X[..., :H * P], H), heads(X[..., H * P:H * P + D], 1), heads(X[..., H * P + D:], 1), dt.reshape(n, -1),
                                        (-torch.exp(a_log.to(F64)) * dt).reshape(n, -1), skip.to(F64).repeat(B), S0)
        else:
            la = -torch.exp(a_log.to(F64)) * torch.nn.functional.softplus(u[..., H:] + bias.to(F64))
            y, S = _delta_reference(heads(X[..., :G * D], G), heads(X[..., G * D:2 * G * D], G), heads(X[..., 2 * G * D:], H),
                                    torch.sigmoid(u[..., :H]).reshape(n, -1), la.reshape(n, -1), S0)
        y, S = y.view(n, B, H, P).transpose(0, 1), S.view(B, H, D, P)
        err = lambda a, b: ((a.to(F64) - b).norm() / b.norm()).item()
        totals += torch.tensor([err(out, y), err(torch.cat(walked, 1), y), err(state, S), err(walked_state, S)], dtype=F64)
    chunk, walk, chunk_state, walk_state = (totals / 8).tolist()
    assert chunk <= walk and chunk_state <= walk_state and max(chunk, chunk_state) < 1.5e-7, (chunk, walk, chunk_state, walk_state)
