"""A wait that ran out inside a kernel reaches the caller of an engine's step (CPU: the runner and the library are stand-ins)."""
from types import SimpleNamespace

import pytest
import torch

import nano_qwen3tts_vllm_b200._native as nat
from nano_qwen3tts_vllm_b200.engine.llm_engine.lm_engine import CausalLMEngine


class _Seq(SimpleNamespace):
    def __len__(self):
        return self.num_tokens


@pytest.mark.parametrize("lost", [False, True])
def test_no_token_is_handed_out_behind_a_wait_that_ran_out(monkeypatch, lost):
    done = []
    engine = CausalLMEngine.__new__(CausalLMEngine)
    seq = _Seq(hold=False, num_cached_tokens=0, num_tokens=3, request_id="a", seq_id=0, top_k=1, temperature=1.0, is_finished=False)
    engine.config = SimpleNamespace(max_model_len=10)
    engine.scheduler = SimpleNamespace(schedule=lambda: [(seq, 3)], postprocess=lambda seqs, tokens: done.extend(tokens))
    engine.model_runner = SimpleNamespace(call=lambda name, *a: torch.zeros(1, 5) if name == "run_step" else torch.tensor([4]))
    library = SimpleNamespace(b2tts_grouped_gemm_check=lambda: 3 if lost else 0, b2tts_last_error=lambda: b"a wait ran out")
    monkeypatch.setattr(nat, "_load", lambda: library)
    if lost:
        with pytest.raises(RuntimeError, match="ran out"):
            engine.step()
    else:
        engine.step()
    assert done == ([] if lost else [4])


@pytest.fixture(params=[False, True], ids=["healthy", "lost"])
def lost(request, monkeypatch):
    """The library's word on its waits; nothing else of it is called here."""
    library = SimpleNamespace(b2tts_grouped_gemm_check=lambda: 3 if request.param else 0, b2tts_last_error=lambda: b"a wait ran out")
    monkeypatch.setattr(nat, "_load", lambda: library)
    return request.param


def _refused_if(lost, call):
    if lost:
        with pytest.raises(RuntimeError, match="ran out"):
            call()
        return None
    return call()


class _Event:
    waited = False

    def synchronize(self):
        self.waited = True


@pytest.mark.parametrize("split", [False, True], ids=["step", "launch_and_collect"])
def test_a_talker_step_hands_out_no_token_behind_a_wait_that_ran_out(lost, split):
    """Prompts replayed from a graph pass no launch's own check: what the step collects behind its synchronisation is checked there."""
    from nano_qwen3tts_vllm_b200.engine.llm_engine.talker_llm_engine import TalkerLLMEngine
    from nano_qwen3tts_vllm_b200.engine.model_runner.talker_mode_runner import TalkerModeModelRunner
    done, event = [], _Event()
    runner = TalkerModeModelRunner.__new__(TalkerModeModelRunner)
    runner.run_launch = lambda seqs, is_prefill: (torch.tensor([7]), event, torch.zeros(1, 2))
    engine = TalkerLLMEngine.__new__(TalkerLLMEngine)
    engine.model_runner = runner
    seq = _Seq(num_tokens=130, is_finished=False, request_id="a", seq_id=0, completion_token_ids=[], last_hidden_state=None)
    engine.scheduler = SimpleNamespace(schedule=lambda: ([seq], True), postprocess=lambda seqs, tokens, hidden: done.extend(tokens))
    _refused_if(lost, (lambda: engine.step_collect(engine.step_launch())) if split else engine.step)
    assert event.waited and done == ([] if lost else [7])


def test_the_predictor_hands_out_no_code_behind_a_wait_that_ran_out(lost):
    from nano_qwen3tts_vllm_b200.engine.llm_engine.predictor_llm_engine import PredictorLLMEngine
    engine = PredictorLLMEngine.__new__(PredictorLLMEngine)
    seq = SimpleNamespace(token_ids=[], last_token=None, request_id="a", seq_id=0, completion_token_ids=[])
    _refused_if(lost, lambda: engine._burst_collect(([seq], torch.tensor([[5, 6]]), _Event())))
    assert seq.token_ids == ([] if lost else [5, 6])
    seq = SimpleNamespace(token_ids=[engine.PENDING], last_token=None, _deferred=[(0, 0)])
    engine._steps = [torch.tensor([9])]
    _refused_if(lost, lambda: engine._resolve([seq]))
    assert seq.token_ids == [engine.PENDING if lost else 9]


def test_the_device_frame_loop_hands_out_no_frame_behind_a_wait_that_ran_out(lost):
    from nano_qwen3tts_vllm_b200.engine.frame_loop import DeviceFrameLoop
    loop = DeviceFrameLoop.__new__(DeviceFrameLoop)
    loop.frame_idx, loop.frames, loop.frames_done = torch.tensor([2]), torch.arange(12).view(3, 2, 2), torch.tensor([2, 1])
    frames, counts = _refused_if(lost, loop.result), _refused_if(lost, loop.frame_counts)
    assert lost or (frames.tolist() == [[[0, 1], [2, 3]], [[4, 5], [6, 7]]] and counts == [2, 1])
