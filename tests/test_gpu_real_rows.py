"""The real-space product from rows shared by four beads, at bead counts that
leave the last group part full and on both sides of the rules that give a group
one, two or four warps, single and blocks of vectors, against
oracle/pme_oracle.py's product with the same discretisation (FP64 1e-11, FP32
storage 1e-5, the bounds of the product's other tests)."""
import numpy as np
import pytest

import bd_b200 as B
import oracle as O
import pme_oracle as P
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 1e-5)])
@pytest.mark.parametrize("N", [1, 61, 3551, 3553, 7103, 7106])
def test_rows_match_model(N, precision, tol):
    L, K, p, rc, alpha, t = max(24.0, (N / 0.05) ** (1 / 3)), 32, 6, 6.0, 0.45, 2000
    r = np.random.default_rng(N)
    x, y, z = (np.ascontiguousarray(v) for v in r.uniform(-L / 2, L / 2, (3, N)))
    o = O.Oracle(0, N, 1, L, 0.2, 5e-4)
    c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_order=p, pme_rc=rc,
                                pme_alpha=alpha, noise_block=8))
    o.lattice(t)
    o.apply_pbc(x, y, z)
    c.set_positions(x, y, z)
    c.set_time(t, t)
    c.update_lattice(t)
    c.calc_hi()
    pos, H = np.stack([x, y, z], 1), P.reduced_cell(list(o.s.L1), list(o.s.L2), L)
    V = r.normal(size=(3, N, 3))
    ar = P.ref_alpha(t, o.s.tp, o.s.L2yp)
    ref = [P.pme_apply(H, pos, V[k], K, p, alpha, rc, alpha_ref=ar).reshape(-1) for k in (0, 2)]
    got = c.mobility_apply_block(V.reshape(3, -1))
    assert rel_err(got[0], ref[0]) < tol
    assert rel_err(got[2], ref[1]) < tol
    assert rel_err(c.mobility_apply(V[0].reshape(-1)), ref[0]) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("N", [7103, 11843, 23685])
def test_blocks_of_nine_match_singles(N, precision, tol):
    """Five packed pairs on the sides of their own rules, against one product per
    vector (the bounds of the block product's other test)."""
    L = (N / 0.05) ** (1 / 3)
    r = np.random.default_rng(N)
    c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=40, pme_rc=6.0, pme_alpha=0.45,
                                noise_block=10))
    c.set_positions(*r.uniform(-L / 2, L / 2, (3, N)))
    c.set_time(0, 0)
    c.update_lattice(0)
    c.apply_pbc()
    c.calc_hi()
    V = r.normal(size=(9, 3 * N))
    got = c.mobility_apply_block(V)
    assert max(rel_err(got[k], c.mobility_apply(V[k])) for k in range(9)) < tol
