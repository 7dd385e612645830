"""Prompt portions of the recurrences with what their keys and queries alone say formed ahead of the chain of chunks: the same numbers, to the
bit, as formed inside it - chunk edges, several portions that share a chunk of rows, carried states, groups, and values out of the split's range
(whose chunks are walked token by token)."""
import pytest
import torch

from tests.lm_util import Lay as StepLay

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SEQS = [[(0, 130)], [(9, 65), (0, 64), (5, 1), (0, 200), (0, 0), (3, 7), (0, 66)], [(0, 63), (0, 63), (0, 63), (700, 321)]]


def _layout(seqs):
    return StepLay([(c, n, list(range(20))) for c, n in seqs], 64, 20)


def _both(run, state):
    got = []
    for ahead in (True, False):
        s = state.clone()
        got.append((run(s, ahead), s))
    (a, sa), (b, sb) = got
    same = lambda x, y: torch.equal(torch.nan_to_num(x, 1.5), torch.nan_to_num(y, 1.5)) and torch.equal(x.isnan(), y.isnan())
    assert same(a, b) and same(sa, sb)
    assert not torch.equal(sa, state)


@pytest.mark.parametrize("seqs", SEQS)
@pytest.mark.parametrize("big", [None, "q", "k", "v"])
@pytest.mark.parametrize("N,H,G", [(128, 8, 2), (64, 4, 1)])
def test_state_space(seqs, big, N, H, G):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator(device=DEV).manual_seed(N + len(seqs))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay, P = _layout(seqs), 64
    n = lay.n_tokens
    x, dt = r(n, H * P + 2 * G * N).bfloat16(), r(n, H).bfloat16()
    if big:
        x[n // 2, {"v": 3, "k": H * P + 5, "q": H * P + G * N + N // 2}[big]] = float("inf") if big == "v" else 1e30
    args, out = (r(H), 0.5 * r(H) - 0.5, r(H)), torch.empty(n, H * P, device=DEV)
    _both(lambda s, ahead: (nat.ssm_scan(x, dt, *args, s, out.fill_(7), lay, H, G, P, N, ahead=ahead), out.clone())[1], r(len(seqs), H, N, P))


@pytest.mark.parametrize("seqs", SEQS)
@pytest.mark.parametrize("big", [None, "q", "k", "v"])
@pytest.mark.parametrize("d,dv,H,G", [(128, 64, 4, 2), (64, 128, 2, 2)])
def test_delta_rule(seqs, big, d, dv, H, G):
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator(device=DEV).manual_seed(d + len(seqs))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay = _layout(seqs)
    n = lay.n_tokens
    x, ba = r(n, 2 * G * d + H * dv).bfloat16(), r(n, 2 * H).bfloat16()
    if big:
        x[n // 2, {"q": 5, "k": G * d + d, "v": 2 * G * d + 3}[big]] = 1e30
    args, out = (0.5 * r(H) - 0.5, r(H)), torch.empty(n, H * dv, device=DEV)
    _both(lambda s, ahead: (nat.delta_rule_scan(x, ba[:, :H], ba[:, H:], *args, s, out.fill_(7), lay, H, G, d, dv, ahead=ahead), out.clone())[1],
          r(len(seqs), H, d, dv))


def _out_of_order(seqs, order):
    """The same rows, described sequence by sequence in another order: starts no longer ascend."""
    lay = _layout(seqs)
    p = torch.tensor(order, device=DEV)
    for name in ("seq_start", "seq_pos0", "seq_len", "seq_slot", "block_tables"):
        setattr(lay, name, getattr(lay, name)[p].contiguous())
    lay.tok_seq = torch.argsort(p)[lay.tok_seq.long()].to(torch.int32)
    return lay


@pytest.mark.parametrize("seqs,order", [([(0, 512), (0, 512)], [1, 0]), ([(9, 64), (0, 64), (0, 0), (5, 320), (0, 200)], [3, 2, 0, 4, 1])])
def test_rows_that_do_not_lie_in_the_order_of_the_sequences(seqs, order):
    """Chunks of two sequences must not share a place in the scratch (chunk 8 of one was the last of the other)."""
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator(device=DEV).manual_seed(len(seqs))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    lay, H, G, d = _out_of_order(seqs, order), 4, 1, 64
    n = lay.n_tokens
    x, dt, args, out = r(n, H * d + 2 * G * d).bfloat16(), r(n, H).bfloat16(), (r(H), 0.5 * r(H) - 0.5, r(H)), torch.empty(n, H * d, device=DEV)
    _both(lambda s, ahead: (nat.ssm_scan(x, dt, *args, s, out.fill_(7), lay, H, G, d, d, ahead=ahead), out.clone())[1], r(len(seqs), H, d, d))
    x, ba, args = r(n, 2 * G * d + H * d).bfloat16(), r(n, 2 * H).bfloat16(), (0.5 * r(H) - 0.5, r(H))
    _both(lambda s, ahead: (nat.delta_rule_scan(x, ba[:, :H], ba[:, H:], *args, s, out.fill_(7), lay, H, G, d, d, ahead=ahead), out.clone())[1],
          r(len(seqs), H, d, d))


@pytest.mark.parametrize("lens", [[200] + [0] * 99, [0] * 40 + [130] + [0] * 30 + [70, 1]])
def test_portions_of_unknown_length_beside_empty_sequences(lens):
    """Without max_new the longest portion is not n_tokens - n_seqs + 1: empty sequences need no row."""
    import nano_qwen3tts_vllm_b200._native as nat
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    n, b, H, d, L, st = sum(lens), len(lens), 4, 64, nat.lib(), torch.cuda.current_stream().cuda_stream
    seq = [i32([sum(lens[:i]) for i in range(b)]), i32([0] * b), i32(lens), i32(list(range(b)))]
    ptrs, out, coef = [t.data_ptr() for t in seq], torch.empty(n, H * d, device=DEV), torch.empty(n, H, 3, device=DEV)
    x, dt, par = r(n, H * d + 2 * d).bfloat16(), r(n, H).bfloat16(), (r(H), 0.5 * r(H) - 0.5, r(H))
    y, ba, par2 = r(n, 2 * d + H * d).bfloat16(), r(n, 2 * H).bfloat16(), (0.5 * r(H) - 0.5, r(H))

    def ssm(s, ahead):
        room = torch.full((L.b2tts_ssm_scan_ahead_floats(n, b, 1),), 3.0, device=DEV)
        assert L.b2tts_ssm_scan_ahead(x.data_ptr(), x.stride(0), dt.data_ptr(), H, *[t.data_ptr() for t in par], s.data_ptr(), coef.data_ptr(),
                                      out.fill_(7).data_ptr(), *ptrs, n, b, 0, H, 1, d, d, nat.DTYPE_CODE[torch.bfloat16],
                                      room.data_ptr() if ahead else None, room.numel(), st) == 0
        return out.clone()

    def delta(s, ahead):
        room = torch.full((L.b2tts_delta_rule_scan_ahead_floats(n, b, 1),), 3.0, device=DEV)
        assert L.b2tts_delta_rule_scan_ahead(y.data_ptr(), y.stride(0), ba.data_ptr(), ba[:, H:].data_ptr(), 2 * H, *[t.data_ptr() for t in par2],
                                             s.data_ptr(), coef.data_ptr(), out.fill_(7).data_ptr(), *ptrs, n, b, 0, H, 1, d, d,
                                             nat.DTYPE_CODE[torch.bfloat16], room.data_ptr() if ahead else None, room.numel(), st) == 0
        return out.clone()
    _both(ssm, r(b, H, d, d))
    _both(delta, r(b, H, d, d))
