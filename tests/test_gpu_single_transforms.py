"""Single products on both sides of the rule that sends them through real
transforms, next to blocks on the same context.  Against oracle/pme_oracle.py (FP64 1e-11, FP32 2e-6, as the other sizes)."""
import functools

import numpy as np
import pytest

import bd_b200 as B
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


@pytest.mark.parametrize("precision,K", [("fp64", 96), ("fp64", 100), ("fp64", 135), ("fp32", 120),
                                         ("fp32", 128), ("fp32", 144), ("fp32", 150)])
@pytest.mark.parametrize("block", [1, 2, 3])
def test_single_products(K, precision, block):
    pos, V, ref = _model(60, K, 8, 3)
    c, tol = _context(pos, K, 8, precision, block)
    first = c.mobility_apply(V[0])
    assert rel_err(first, ref[0]) < tol
    if block > 1:  # a block on the same grids in between
        got = c.mobility_apply_block(V[:block])
        assert max(rel_err(got[r], ref[r]) for r in range(block)) < tol
    assert np.array_equal(c.mobility_apply(V[0]), first)
