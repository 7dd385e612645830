"""Decode attention in one launch over head counts: every instance that is chosen by query heads a key head and by key heads, with and without splits, against the separate
launches, and against sums cut into other splits."""
import pytest
import torch

from . import test_gpu_fused_attn as one

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (2, 2), (8, 8), (2, 1), (4, 2), (6, 3), (8, 4), (10, 5), (16, 8), (4, 1), (8, 2), (12, 3), (16, 4), (20, 5), (32, 8)])
@pytest.mark.parametrize("b,max_len,room", [(3, 40, None), (40, 300, None), (5, 1000, 4096), (300, 70, None)])
def test_head_counts(native, monkeypatch, heads, kv_heads, b, max_len, room):
    monkeypatch.setattr(one, "H", heads)
    monkeypatch.setattr(one, "KVH", kv_heads)
    for rounding in (native.ROUND_EAGER, native.ROUND_FUSED):
        one._case(native, b, max_len, mrope=kv_heads % 2 == 0, rounding=rounding, seed=b + heads, pad_rows=min(1, b - 2), max_ctx_override=room)
