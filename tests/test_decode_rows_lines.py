"""Which decode steps of a few rows the persistent kernel takes (csrc/decode_rows.cu): by rows and by the room that the tables have for a context, up to where a CTA of
attention would have to walk its splits in turns.  On 148 multiprocessors (as the library assumes where there is no GPU)."""
import ctypes

import pytest
import torch

from nano_qwen3tts_vllm_b200 import _native as nat

TALKER, SMALL = (2048, 2048, 1024, 6144), (1024, 2048, 1024, 3072)


@pytest.mark.parametrize("widths,rows,most", [(TALKER, 1, 10 ** 6), (TALKER, 2, 10 ** 6), (TALKER, 3, 1592), (TALKER, 4, 1080), (TALKER, 5, 0), (SMALL, 1, 10 ** 6), (SMALL, 2, 10 ** 6),
                                             (SMALL, 3, 1592), (SMALL, 4, 1080), (SMALL, 5, 824), (SMALL, 6, 824), (SMALL, 7, 568), (SMALL, 8, 568), (SMALL, 9, 0)])
def test_room_for_contexts(widths, rows, most):
    for room in (1, 32, 256, 568, 569, 824, 825, 1080, 1081, 1592, 1593, 2048, 4096, 32768):
        assert nat.decode_rows_taken(rows, room, *widths) == (room <= most), room
    assert not nat.decode_rows_taken(rows, 0, *widths)


def test_widths_without_a_kernel():
    for widths in [(1024, 2048, 512, 3072), (2560, 2048, 1024, 9728), (512, 1024, 512, 1536)]:
        assert not any(nat.decode_rows_supported(m, *widths) or nat.decode_rows_taken(m, 32, *widths) for m in range(1, 9))


@pytest.mark.parametrize("page", [1, 2, 4, 12, 24, 100, 8, 256])
def test_pages_that_the_separate_launches_refuse(page):
    """Pages that do not hold whole tiles of eight tokens are refused as by fused_decode_attn; others fail at the next check only (of the workspace: nothing is launched)."""
    keep = torch.zeros(64, dtype=torch.uint8)
    at = (keep.data_ptr() + 15) // 16 * 16
    layers = nat.stack_layer_array([{n: torch.zeros(16, dtype=torch.bfloat16) for n in ("qkv_w", "o_w", "gate_up_w", "down_w", "input_norm_w", "post_norm_w", "q_norm_w", "k_norm_w",
                                                                                       "k_cache", "v_cache")}])
    lib = nat.lib()
    rc = lib.b2tts_decode_rows(at, 1024, at, 1024, ctypes.byref(layers), 1, at, 1, 1024, 16, 8, 128, 3072, 1e-6, 0, at, 0, at, None, 1.0, at, at, 1, at, page, 64, 0.1, 256, 0, None)
    said = lib.b2tts_last_error().decode()
    assert rc != 0 and ("pages of" in said) == (page not in (8, 256)) and ("workspace" in said) == (page in (8, 256)), said
