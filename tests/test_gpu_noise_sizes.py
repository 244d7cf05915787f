"""The reference's ran1/gasdev stream drawn by a warp: every draw count around
the batches of 32 pairs (a draw's last deviate may fall anywhere in a batch,
and an odd count leaves one deviate for the next draw), from the seed on and
over several draws, bit for bit against oracle/bd_oracle.c, the generator's
state included."""
import ctypes as C

import numpy as np
import pytest

import bd_b200 as B
import oracle as O

pytestmark = pytest.mark.gpu


def _context(n, seed):
    return B.Context(B.make_params(0, n, 1, 30.0, 0.1, 5e-4, noise="ran1", seed=seed))


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 15, 16, 17, 21, 33, 50, 67, 128, 500])
@pytest.mark.parametrize("seed", [830062920, -12345, 981272199])
def test_stream_matches_oracle(n, seed):
    c = _context(n, seed)
    rng = O.fresh_rng(seed)
    R = np.zeros(3 * n)
    for _ in range(5):
        c.get_noise()
        O.lib().bdo_noise(C.byref(rng), R, 3 * n)
        assert np.array_equal(c.noise(), R)
        assert np.array_equal(c.rng().state_words(), rng.state_words())
