"""Grid sizes whose transforms go through cuFFT: components one after the other, real
transforms for a single right-hand side, packed pairs otherwise, odd last ones
among them, in a skewed cell, against oracle/pme_oracle.py (FP64 1e-11, FP32 2e-6 as
for the other sizes)."""
import functools

import numpy as np
import pytest

import bd_b200 as B
import oracle as O
import pme_oracle as P
from conftest import rel_err

pytestmark = pytest.mark.gpu

NB, NC, L, T = 20, 3, 24.0, 3000
ALPHA, RC = 0.35, 10.0


@functools.lru_cache(maxsize=None)
def _model(K, p, flow):
    x, y, z = B.random_chains(NB, NC, L, 23, bond=2.0, min_sep=1.8)
    x, y = B.lab_frame(flow, x, y)
    o = O.Oracle(flow, NB, NC, L, 0.2, 5e-4)
    o.lattice(T)
    if flow == 1:
        o.rotate(x, y, 0)
    o.apply_pbc(x, y, z)
    xl, yl = (x * o.s.cth - y * o.s.sth, x * o.s.sth + y * o.s.cth) if flow else (x, y)
    H = P.reduced_cell(list(o.s.L1), list(o.s.L2), L)
    V = np.random.default_rng(K).normal(size=(5, NB * NC, 3))
    ar = P.ref_alpha(T, o.s.tp, o.s.L2yp)
    pos = np.stack([xl, yl, z], 1)
    ref = [P.pme_apply(H, pos, v, K, p, ALPHA, RC, alpha_ref=ar).reshape(-1) for v in V]
    return (x, y, z), V.reshape(5, -1), np.stack(ref)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-6)])
@pytest.mark.parametrize("block", [1, 5])
@pytest.mark.parametrize("K,p,flow", [(8, 4, 0), (13, 6, 1), (22, 8, 0), (35, 4, 1), (49, 6, 0),
                                      (70, 8, 1), (125, 8, 1), (125, 6, 0)])
def test_planar_grids_match_model(K, p, flow, block, precision, tol):
    pos, V, ref = _model(K, p, flow)
    c = B.Context(B.make_params(flow, NB, NC, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_order=p, pme_rc=RC,
                                pme_alpha=ALPHA, noise_block=block))
    c.set_positions(*pos)
    c.set_time(T, T)
    c.update_lattice(T)
    c.calc_hi()
    assert rel_err(c.mobility_apply(V[0]), ref[0]) < tol
    for k in (2, 5) if block > 1 else ():
        got = c.mobility_apply_block(V[:k])
        assert max(rel_err(got[r], ref[r]) for r in range(k)) < tol
    assert rel_err(c.mobility_apply(V[1]), ref[1]) < tol
