"""8-bit-slice launches of hundreds of small problems, whose operand sides are
looked up by address: shared and unshared sides of instances of many sizes."""
import pytest

import test_i8_tiles_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(12, 17 + j, j % 3) for j in range(16)], [(60, 20, 2)], [(1, 1, 1)]])
def test_grouped_selected_inversion_of_many_blocks(sizes, monkeypatch):
    base.test_grouped_selected_inversion(sizes, 0, monkeypatch)
