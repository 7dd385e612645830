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
