"""Sweeps through block inverses with large products: blocks wider than the 4096
vector entries that are staged at a time, whose strips from column 4096 on are
the first of a CTA's share (from b = 4113 on with one CTA per SM), alone and
beside a smaller instance; and steps of more than 64 MB, whose rows are dealt
in pairs."""
import numpy as np
import pytest

import test_sweep_inv_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cand", range(2))
@pytest.mark.parametrize("sizes", [[(2, 4500, 3)], [(1, 5025, 0)], [(2, 4500, 0), (2, 4500, 1)],
                                   [(3, 130, 0), (2, 4500, 3)], [(1, 8210, 2)]])
def test_wide_blocks_solve_with_the_factor(sizes, cand, monkeypatch):
    base.test_sweeps_solve_with_the_factor(sizes, cand, monkeypatch)


# a step's larger product has more than 64 MB: rows in pairs, odd and even b, an instance of few rows among them
@pytest.mark.parametrize("cand", range(2))
@pytest.mark.parametrize("sizes", [[(2, 2900, 3)], [(2, 1999, 2), (1, 65, 1), (3, 2500, 0)], [(1, 4095, 0)],
                                   [(2, 517, 1)] * 33])
def test_large_products_solve_with_the_factor(sizes, cand, monkeypatch):
    base.test_sweeps_solve_with_the_factor(sizes, cand, monkeypatch)


def test_wide_model_mean_agrees_with_the_tile_sweep():
    """f and the latent mean by block inverses (``evaluate_f``, the gradient's
    forward half) and by the tile sweep (the batched f of this width)."""
    import torch

    from dalia_b200 import synth
    from dalia_b200.model import SpatioTemporalModel

    theta = np.array([-1.0, 1.0, 0.0, 2.0])
    m = SpatioTemporalModel(synth.make_problem(4489, 3, 2, 300, theta))
    f_tile = m.evaluate_f_batched([theta])[0]
    x_tile = m.x.clone()
    f_inv = m.evaluate_f(theta)
    # both solve with one factor: they differ by condition number x rounding, some 1e-9 here at most;
    # 16 columns lost out of 4489 change the mean by 1e-2
    assert abs(f_inv - f_tile) <= 1e-9 * abs(f_tile)
    assert float((m.x - x_tile).norm() / x_tile.norm()) <= 1e-7
    m.adjoint_forward([theta])
    assert float((m.slots[0].x - x_tile).norm() / x_tile.norm()) <= 1e-7
    assert bool(torch.isfinite(m.x).all())
