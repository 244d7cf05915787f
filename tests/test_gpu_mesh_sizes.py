"""Spreading, transforms and interpolation of the particle-mesh product over
grid sizes, spline orders and numbers of right-hand sides: sizes of every pair
of transform factors up to 150, odd ones, sizes that fall through to cuFFT (a
factor 7, 11, 13, or below 20), columns cut short at the grid's edge (sizes not
divisible by 2, 3, 4, 5, 8), and each number of packed pairs that has a column
layout of its own, an odd last right-hand side among them.

Against oracle/pme_oracle.py (same grid, order, split, cutoff).  FP64 1e-11,
the bound of the existing comparison with that model; FP32 2e-6: weights,
grids, transforms and pair terms hold 24 bits (6e-8 each), a result adds some
tens of such roundings of terms a few times its own size."""
import numpy as np
import pytest

import bd_b200 as B
import pme_oracle as P
from conftest import rel_err

pytestmark = pytest.mark.gpu

NB, NC, L = 10, 6, 24.0


def _context(K, p, precision, k):
    x, y, z = B.random_chains(NB, NC, L, 17, bond=2.0, min_sep=1.8)
    c = B.Context(B.make_params(0, NB, NC, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_order=p, pme_rc=10.0,
                                pme_alpha=0.35, noise_block=k))
    c.set_positions(x, y, z)
    c.set_time(0, 0)
    c.update_lattice(0)
    c.calc_hi()
    return c, np.stack([x, y, z], 1)


def _check(K, p, precision, k):
    c, pos = _context(K, p, precision, k)
    V = np.random.default_rng(K + k).normal(size=(k, 3 * NB * NC))
    got = c.mobility_apply_block(V)
    again = c.mobility_apply_block(V)
    H = P.cell([L, 0.0], [0.0, L], L)
    ref = np.stack([P.pme_apply(H, pos, v.reshape(-1, 3), K, p, 0.35, 10.0,
                                alpha_ref=4.0 / L).reshape(-1) for v in V])
    assert rel_err(got, ref) < (1e-11 if precision == "fp64" else 2e-6)
    assert np.array_equal(got, again)  # sums in a fixed order


SIZES = [8, 13, 18, 20, 21, 22, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81,
         90, 96, 100]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("K", SIZES)
def test_grid_sizes(K, precision):
    _check(K, 8, precision, 3)


@pytest.mark.parametrize("K", [108, 120, 128, 135, 144, 150])
def test_large_grid_sizes(K):
    _check(K, 8, "fp32", 2)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [4, 6, 8])
@pytest.mark.parametrize("k", [1, 2, 4, 5, 7, 10, 13])
def test_right_hand_sides_and_orders(k, p, precision):
    _check(27, p, precision, k)
