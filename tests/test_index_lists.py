"""Index and scalar lists of the binding: what is kept between calls depends on the numbers alone."""
import numpy as np
import pytest
import torch

from cerium_b200 import _capi


@pytest.mark.parametrize("convert", [_capi._u32, _capi._u64])
def test_lists_are_converted_by_value(convert):
    boxes = [torch.tensor(3), torch.tensor(5)]          # hashed by identity, changed in place
    assert list(convert(boxes)) == [3, 5]
    boxes[0].fill_(4)
    assert list(convert(boxes)) == [4, 5]
    cells = [np.array(3), np.array(5)]                  # not hashable
    assert list(convert(cells)) == [3, 5]
    cells[1][...] = 6
    assert list(convert(cells)) == [3, 6]
    index = np.array([7, 8], dtype=np.int64)
    assert list(convert(index)) == [7, 8]
    index[0] = 9
    assert list(convert(index)) == [9, 8]
    assert list(convert([2.0, True])) == [2, 1] and list(convert(range(3))) == [0, 1, 2] and list(convert([])) == []
    with pytest.raises((TypeError, ValueError)):
        convert(["a"])
