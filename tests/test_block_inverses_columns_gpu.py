"""Inverses of many lower-triangular blocks, a CTA per tile column: on both sides
of the rule that chooses it (b = 130 from 320 blocks on, with three CTAs on each
of 148 SMs), odd row strides, and instances of one to five tiles a row in one
launch."""
import pytest

import test_block_inverses_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(319, 130)], [(320, 130)], [(210, 321)], [(90, 577)],
                                   [(400, 257), (3, 130), (30, 64), (100, 300)], [(5, 1)] * 66 + [(500, 192)]])
def test_block_inverses_by_columns(sizes):
    base.test_block_inverses_at_tile_edges(sizes)
