"""What a step's layout tells the kernels' wrappers about its sequences (CPU)."""
from types import SimpleNamespace

import pytest
import torch

from nano_qwen3tts_vllm_b200.engine.step_layout import MixedStepLayout


@pytest.mark.parametrize("items,max_new,max_keys", [
    ([(0, 300)], 300, 300), ([(0, 300), (900, 1), (20, 1)], 300, 300), ([(10, 40), (0, 33), (500, 1)], 40, 50), ([(900, 1), (3, 1)], 1, 0), ([], 0, 0)])
def test_the_longest_portions_keys(items, max_new, max_keys):
    """Decoded tokens beside a portion do not make it a long one: which kernel takes the portions goes by their own keys."""
    seq = lambda c, n: SimpleNamespace(num_cached_tokens=c, block_table=list(range(-(-(c + n) // 16))), token_ids=[1] * (c + n), state_slot=0)
    lay = MixedStepLayout(512, 4, 64, torch.device("cpu"))
    lay.fill([(seq(c, n), n) for c, n in items], 16)
    assert (lay.max_new, lay.max_keys, lay.n_seqs) == (max_new, max_keys, len(items))
    assert lay.portions == items
