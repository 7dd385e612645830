"""The numbers that words carry in the persistent decode step (csrc/decode_rows.cu) run through 2^32: words of steps long ago are not taken for new ones."""
import pytest
import torch

from tests.test_gpu_decode_rows import _case, _stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,layers,rows,lens", [(1024, 3072, 5, 8, 40), (1024, 3072, 5, 2, 2500), (2048, 6144, 3, 4, 100)])
@pytest.mark.parametrize("behind", [0, 1, 7])
def test_numbers_start_anew(hidden, inter, layers, rows, lens, behind):
    stack = _stack(hidden, inter, layers, False, 0)
    stack._rows_ws = None
    first, second = _case(stack, rows, lens, 3), _case(stack, rows, lens, 4)
    want = [run(False) for run in (first, second)]
    same = lambda got, k: torch.equal(got[0], want[k][0]) and all(torch.equal(a, c) and torch.equal(b, d) for (a, b), (c, d) in zip(got[1], want[k][1]))
    assert same(first(True), 0)                                  # numbers 1 ..: from a workspace of zeros
    number = stack._rows_ws[:8].view(torch.int32)
    assert number.tolist() == [8 * layers, 0]
    number[0] = -8 * layers * (behind + 1)                       # so many steps in front of 2^32
    for k in range(behind + 1):
        assert same(second(True), 1)
    # behind one of the last steps every word was cleared, so that the words that the first step left are gone
    assert 0 <= number[0].item() <= 8 * layers * 7 and number[1].item() == 0
    assert same(second(True), 1) and same(first(True), 0)


def test_words_are_cleared():
    stack = _stack(1024, 3072, 5, False, 0)
    stack._rows_ws = None
    run = _case(stack, 8, 2000, 3)
    run(True)
    assert int((stack._rows_ws[256:] != 0).sum()) > 0
    stack._rows_ws[:8].view(torch.int32)[0] = -8 * 5
    run(True)
    assert int((stack._rows_ws != 0).sum()) == 0
