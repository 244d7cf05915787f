"""The square root with vectors orthogonalised by one cluster (up to 2048 beads)
and past it: applied twice it is the mobility.  Solves to 1e-8 (relative change of
the iterate); the bound of 1e-5 leaves the tail estimate and the square a factor of
a thousand."""
import numpy as np
import pytest

import bd_b200 as B
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nb,Nc", [(1, 1), (2, 1), (11, 3), (65, 1), (25, 20), (64, 32), (683, 3)])
def test_square_root_applied_twice_is_the_product(Nb, Nc):
    N = Nb * Nc
    L = max(24.0, (N / 0.05) ** (1 / 3))
    r = np.random.default_rng(N)
    m = int(np.ceil(N ** (1 / 3)))  # jittered lattice, no overlaps needed
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:N]
    x, y, z = np.ascontiguousarray((g * (L / m) + r.uniform(0, 0.3, (N, 3)) - L / 2).T)
    c = B.Context(B.make_params(0, Nb, Nc, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                lanczos_tol=1e-8))
    c.set_positions(x, y, z)
    c.set_time(0, 0)
    c.update_lattice(0)
    c.apply_pbc()
    c.calc_hi()
    v = r.normal(size=3 * N)
    half, it = c.lanczos_sqrt(v)
    twice, _ = c.lanczos_sqrt(half)
    assert it >= 1
    assert rel_err(twice, c.mobility_apply(v)) < 1e-5
