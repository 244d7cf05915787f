"""bd_autotune_pme_grid ranks grid sizes by the transforms that a product runs (its
own for sizes with factors up to 16, cuFFT's for the others): the size it picks is,
by the products of a few beads, near the fastest of its candidates.  The sizes
between 200 and 250 differ by factors of up to two; a quarter is left for noise."""
import numpy as np
import pytest

import bd_b200 as B

pytestmark = pytest.mark.gpu


def _smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


def _product_ms(K, L, precision):
    N = 200
    r = np.random.default_rng(0)
    c = B.Context(B.make_params(0, 50, N // 50, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, noise_block=2))
    c.set_positions(*r.uniform(-L / 2, L / 2, (3, N)))
    c.set_time(0, 0)
    c.update_lattice(0)
    c.calc_hi()
    V, ms = r.normal(size=(2, 3 * N)), []
    for _ in range(12):
        c.profile(1)
        c.mobility_apply_block(V)
        t, n = c.profile_read(0)
        ms.append(t / max(n, 1))
    c.close()
    return float(np.median(ms))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_choice_is_near_the_fastest(precision):
    L = 155.0
    K0 = int(np.ceil(1.29 * L))
    sizes = [K for K in range(K0, int(np.ceil(1.25 * K0)) + 1) if _smooth(K)]
    K = B.autotune_pme_grid(L, precision)
    assert K in sizes
    ms = {k: _product_ms(k, L, precision) for k in sizes}
    assert ms[K] < 1.25 * min(ms.values()), (K, ms)
