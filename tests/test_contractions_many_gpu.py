"""Contractions over many blocks, where a block gets eight, four, two or one
CTAs: both sides of the steps on 148 SMs, and variates beside time steps."""
import pytest

import test_contractions_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,n,nv", [(33, 37, 1), (33, 38, 1), (20, 74, 1), (65, 75, 1), (20, 148, 1), (31, 149, 1),
                                     (9, 102, 1), (9, 103, 1), (5, 204, 1), (5, 410, 1), (9, 20, 3), (3, 700, 1)])
def test_block_contractions_over_many_blocks(ns, n, nv):
    base.test_block_contractions(ns, n, nv, 0)
