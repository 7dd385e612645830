"""Which decode steps go to the persistent kernel (models/qwen3_tts_share.py): the switches that led to other launches lead there still, and it has one of its own (the
library and the stack are stand-ins)."""
from types import SimpleNamespace

import pytest
import torch

import nano_qwen3tts_vllm_b200._native as nat
from nano_qwen3tts_vllm_b200.models import qwen3_tts_share as share
from nano_qwen3tts_vllm_b200.utils.context import reset_context, set_context


@pytest.fixture
def takes(monkeypatch):
    asked = []
    monkeypatch.setattr(nat, "decode_rows_taken", lambda *a: asked.append(a) or True)
    stack = SimpleNamespace(_rows_ws=object(), _rows_most=8, _rows_where_faster=True, layers=[SimpleNamespace(self_attn=SimpleNamespace(attn=SimpleNamespace(
        k_cache=torch.zeros(1, 256, 8, 128))))], _widths=lambda: (1024, 2048, 1024, 3072))
    stack._max_context = lambda: share.DecoderStack._max_context(stack)
    set_context(False, block_tables=torch.zeros(8, 3, dtype=torch.int32), context_lens=torch.ones(8, dtype=torch.int32), slot_mapping=torch.zeros(8, dtype=torch.int32))
    yield lambda m=2, **k: share.DecoderStack._takes_rows(stack, torch.zeros(m, 1024, dtype=torch.bfloat16)), stack, asked
    reset_context()


@pytest.mark.parametrize("name,value,rows", [("DECODE_ROWS_MAX", 0, []), ("DECODE_ROWS_MAX", 3, [1, 2, 3]), ("GEMM_NATIVE_MAX_M", 0, []), ("GEMM_NATIVE_MAX_M", 2, [1, 2]),
                                             ("FUSED_DECODE_ATTENTION", False, []), ("GEMM_CHAIN", True, []), ("FUSED_NORM_MIN_ROWS", 5, [1, 2, 3, 4]),
                                             ("FUSED_NORM_MIN_ROWS", 0, []), (None, None, [1, 2, 3, 4, 5, 6, 7, 8])])
def test_switches(monkeypatch, takes, name, value, rows):
    if name is not None:
        monkeypatch.setattr(share, name, value)
    assert [m for m in range(0, 10) if takes[0](m)] == rows


def test_what_the_library_is_asked(takes):
    take, stack, asked = takes
    assert take(3) and asked == [(3, 768, 1024, 2048, 1024, 3072)]
    set_context(False, block_tables=torch.zeros(8, 3, dtype=torch.int32), max_context_len=17)
    assert take(2) and asked[1][:2] == (2, 17)
    stack._rows_where_faster = False
    assert take(2) and len(asked) == 2
    set_context(True, block_tables=torch.zeros(8, 3, dtype=torch.int32))
    assert not take(2)
