"""The one-warp decode attention of short contexts over its whole range: every number of tiles up to the largest context that takes it, the bits of the streaming kernel."""
import pytest
import torch

from . import test_gpu_fused_attn as one

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_len", [1, 8, 9, 16, 17, 24, 33, 50, 63, 64])
@pytest.mark.parametrize("b,rounding", [(1, 0), (37, 1)])
def test_every_number_of_tiles(native, max_len, b, rounding):
    one.test_short_context_kernel_is_bit_identical(native, b, max_len, rounding, 0)
