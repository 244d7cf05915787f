"""Spreading on both sides of the rule that takes one packed pair a warp where beads
are few for the grid: every number of pairs with a column layout of its own, on a
grid small enough for the beads.  Against oracle/pme_oracle.py (FP64 1e-11, FP32
2e-6, as the other sizes)."""
import functools

import numpy as np
import pytest

import bd_b200 as B
import oracle as O
import pme_oracle as P
from conftest import rel_err

pytestmark = pytest.mark.gpu

L, ALPHA, RC = 24.0, 0.35, 10.0


@functools.lru_cache(maxsize=None)
def _model(N, K, p, k):
    r = np.random.default_rng(N + K + p)
    pos, V = r.uniform(-L / 2, L / 2, (N, 3)), r.normal(size=(k, N, 3))
    H = P.cell([L, 0.0], [0.0, L], L)
    ref = [P.pme_apply(H, pos, v, K, p, ALPHA, RC, alpha_ref=4.0 / L).reshape(-1) for v in V]
    return pos, V.reshape(k, -1), np.stack(ref)


def _context(pos, K, p, precision, block):
    c = B.Context(B.make_params(0, 20, len(pos) // 20, L, 0.2, 5e-4, mobility="pme",
                                noise="philox", precision=precision, pme_grid=K, pme_order=p,
                                pme_rc=RC, pme_alpha=ALPHA, noise_block=block))
    c.set_positions(*(np.ascontiguousarray(a) for a in pos.T))
    c.set_time(0, 0)
    c.update_lattice(0)
    c.calc_hi()
    return c, 1e-11 if precision == "fp64" else 2e-6


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [4, 6, 8])
@pytest.mark.parametrize("k", [2, 4, 5, 7, 10, 13])
def test_layouts_of_dense_grids(k, p, precision):
    pos, V, ref = _model(500, 27, p, 13)
    c, tol = _context(pos, 27, p, precision, k)
    got = c.mobility_apply_block(V[:k])
    assert max(rel_err(got[r], ref[r]) for r in range(k)) < tol
    assert rel_err(c.mobility_apply(V[0]), ref[0]) < tol


@pytest.mark.parametrize("precision,N", [("fp64", 200), ("fp64", 220), ("fp32", 400), ("fp32", 440)])
def test_layouts_at_the_density_rule(N, precision):
    pos, V, ref = _model(N, 30, 8, 5)  # 30^3 = 27000: 211 and 422 beads
    c, tol = _context(pos, 30, 8, precision, 5)
    got = c.mobility_apply_block(V)
    assert max(rel_err(got[r], ref[r]) for r in range(5)) < tol


@functools.lru_cache(maxsize=None)
def _sheared(N, K, t):
    """Positions in a sheared cell, a vector and its product."""
    edge = (N / 0.02) ** (1 / 3)
    r = np.random.default_rng(N)
    x, y, z = (np.ascontiguousarray(v) for v in r.uniform(-edge / 2, edge / 2, (3, N)))
    o = O.Oracle(0, 20, N // 20, edge, 0.2, 5e-4)
    o.lattice(t)
    o.apply_pbc(x, y, z)
    v = r.normal(size=(N, 3))
    ref = P.pme_apply(P.reduced_cell(list(o.s.L1), list(o.s.L2), edge), np.stack([x, y, z], 1), v,
                      K, 8, 0.3, 6.0, alpha_ref=P.ref_alpha(t, o.s.tp, o.s.L2yp))
    return edge, (x, y, z), v.reshape(-1), ref.reshape(-1)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("N,K", [(14000, 96), (60, 100)])
def test_columns_in_one_segment(N, K, precision):
    """Enough columns to fill the chip: each is walked whole, from the wrapped bases
    below its first level to the last; five pairs a warp (14 000 beads) and one."""
    t = 2000
    edge, pos, v, ref = _sheared(N, K, t)
    c = B.Context(B.make_params(0, 20, N // 20, edge, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_rc=6.0, pme_alpha=0.3,
                                noise_block=10))
    c.set_positions(*pos)
    c.set_time(t, t)
    c.update_lattice(t)
    c.calc_hi()
    factors = np.array([1.0, -2.0, 3.0, 0.5, -1.25, 0.75, 2.5, -0.375, 1.5, -0.6])
    got = c.mobility_apply_block(factors[:, None] * v)
    tol = 1e-11 if precision == "fp64" else 2e-6
    assert max(rel_err(got[r], f * ref) for r, f in enumerate(factors)) < tol
