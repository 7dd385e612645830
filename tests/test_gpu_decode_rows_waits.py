"""Waits of the persistent decode step that run out (csrc/decode_rows.cu): the launch ends and says so, once, and the next launch on the same workspace has the right bits."""
import pytest
import torch

from tests.test_gpu_decode_rows import _case, _stack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    import nano_qwen3tts_vllm_b200._native as n
    return n


def _step(stack, rows=2, seed=5):
    return _case(stack, rows, 300, seed)


def test_a_wait_that_ran_out_is_an_error(nat):
    """The next step refuses once, and so does the check that the engines make; the next call after that runs again."""
    stack = _stack(1024, 3072, 5, False, 0)
    run = _step(stack)
    want = run(True)[0]
    before = nat.decode_rows_timeouts()
    for consumer in (lambda: run(True), nat.check_waits):
        assert nat.lib().b2tts_decode_rows_lose_wait(None) == 0
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="decode step ran out"):
            consumer()
        nat.check_waits()
        assert torch.equal(run(True)[0], want)
    assert nat.decode_rows_timeouts() == before + 2


@pytest.mark.parametrize("polls", [0, 1, 3])
@pytest.mark.parametrize("hidden,inter,layers,rows,max_len", [(1024, 3072, 5, 8, 40), (2048, 6144, 3, 1, 1300), (2048, 6144, 28, 4, 100)])
def test_every_wait_of_a_step_runs_out(nat, monkeypatch, hidden, inter, layers, rows, max_len, polls):
    """Waits that give up after a few tries: words take longer than that from one multiprocessor to another, so that CTAs go on without them in every phase."""
    stack = _stack(hidden, inter, layers, False, 0)
    run = _case(stack, rows, max_len, 7)
    want, caches = run(False)
    assert torch.equal(run(True)[0], want)
    head = lambda: stack._rows_ws[:8].view(torch.int32).tolist()
    number, step = head(), layers * 8
    assert number[1] == 0
    plain, before = nat.decode_rows, nat.decode_rows_timeouts()
    for _ in range(3):
        monkeypatch.setattr(nat, "decode_rows", lambda *a, **k: plain(*a, **k, polls=polls))
        with pytest.raises(RuntimeError, match="decode step ran out"):
            run(True)                                            # its own check, behind the launch's end
        monkeypatch.setattr(nat, "decode_rows", plain)
        assert nat.decode_rows_timeouts() > before
        before = nat.decode_rows_timeouts()
        assert head() == [number[0] + step, 0]                   # every CTA came to its end
        again = run(True)
        assert torch.equal(again[0], want)
        assert all(torch.equal(a, b) and torch.equal(c, d) for (a, c), (b, d) in zip(again[1], caches))
        number = head()
