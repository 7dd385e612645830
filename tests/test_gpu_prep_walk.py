"""Attention steps of many tokens, each thread with its piece of the row over a run of tokens: every remainder of a run, heads that leave a warp or a block of pieces
partly empty, both pairings and no rotation, tied values."""
import pytest

from .test_gpu_attn_prep import test_against_64_bits as _against_64_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", list(range(1186, 1192)))
@pytest.mark.parametrize("head_norm,norm,rot,interleaved,tied,d,dv", [
    (True, True, 128, True, False, 128, 24), (True, True, 64, False, False, 64, 64), (True, False, 32, False, False, 32, 8), (True, True, 0, True, False, 256, 128),
    (True, False, 16, True, False, 256, 256), (False, False, 0, True, True, 64, 64)])
def test_remainders_of_a_run(n, head_norm, norm, rot, interleaved, tied, d, dv):
    _against_64_bits(n, head_norm, norm, rot, interleaved, tied, d, dv)
