"""Which steps of the delta rule form what their chunks say without the state ahead of the chain, and that steps on either side of those lines give the same bits: few
short portions and many of them, and steps whose scratch would be more than there is to be."""
import pytest
import torch

from tests.test_gpu_scan_chunk import Lay

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(nat, monkeypatch, lens, H, G, D, P, ahead=None):
    """(outputs, state, floats of scratch that the call was given)"""
    g = torch.Generator(device=DEV).manual_seed(sum(lens))
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    n, lay, got = sum(lens), Lay([(5, m, i) for i, m in enumerate(lens)]), []
    lay.max_new = max(lens)
    x, ba = r(n, 2 * G * D + H * P).bfloat16(), r(n, 2 * H).bfloat16()
    a_log, bias, state, out = 0.5 * r(H) - 0.5, r(H), r(len(lens), H, D, P), torch.empty(n, H * P, device=DEV)
    lib = nat.lib()

    class Spy:
        def __getattr__(self, name):
            f = getattr(lib, name)
            if name != "b2tts_delta_rule_scan_ahead":
                return f
            return lambda *a: (got.append(a[-2]), f(*a))[1]
    with monkeypatch.context() as m:
        m.setattr(nat, "_load", lambda: Spy())
        nat.delta_rule_scan(x, ba[:, :H], ba[:, H:], a_log, bias, state, out, lay, H, G, D, P, ahead=ahead)
    return out, state, got[0]


@pytest.mark.parametrize("lens,taken", [([64], False), ([65], False), ([130, 20], False), ([192] * 4, False), ([193], True), ([65] * 5, True), ([100] * 4, False), ([100] * 5, True),
                                        ([100] + [1] * 63, False)])
def test_lines(monkeypatch, lens, taken):
    import nano_qwen3tts_vllm_b200._native as nat
    assert nat.device_info()["sm_count"] == 148                  # what the cases were made for
    out, state, room = _step(nat, monkeypatch, lens, 16, 8, 128, 128)
    assert (room > 0) == taken
    for ahead in (True, False):
        out2, state2, room2 = _step(nat, monkeypatch, lens, 16, 8, 128, 128, ahead=ahead)
        assert (room2 > 0) == (ahead and max(lens) > 64) and torch.equal(out, out2) and torch.equal(state, state2)


@pytest.mark.parametrize("lens", [[300, 70], [100] * 9])
def test_steps_that_would_need_too_much_scratch(monkeypatch, lens):
    import nano_qwen3tts_vllm_b200._native as nat
    out, state, room = _step(nat, monkeypatch, lens, 16, 8, 64, 128)
    assert room > 0
    monkeypatch.setattr(nat, "DELTA_SCRATCH_MOST", room)
    assert _step(nat, monkeypatch, lens, 16, 8, 64, 128)[2] == room
    monkeypatch.setattr(nat, "DELTA_SCRATCH_MOST", room - 1)
    out2, state2, room2 = _step(nat, monkeypatch, lens, 16, 8, 64, 128)
    assert room2 == 0 and torch.equal(out, out2) and torch.equal(state, state2)
