"""Device memory that runs out: a call whose buffers cannot be had returns an
error status, leaves the context without a mobility (products are refused, not
run on missing buffers), fails the same way when it is called again, and works
once there is memory.  The memory is filled through torch; 4000 beads within a
few radii of each other need rows of 4000 entries, 140 MB and more."""
import gc

import numpy as np
import pytest
import torch

import bd_b200 as B

pytestmark = pytest.mark.gpu

N, L = 4000, 60.0
OOM, STATE = 3, 8  # BD_ERR_OOM, BD_ERR_STATE


def _context(precision, block):
    c = B.Context(B.make_params(0, 50, N // 50, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, noise_block=block, pme_rc=12.0))
    c.set_time(0, 0)
    c.update_lattice(0)
    return c


def _spread(c, seed=1):
    c.set_positions(*np.random.default_rng(seed).uniform(-L / 2, L / 2, (3, N)))


def _condense(c):
    c.set_positions(*np.random.default_rng(2).uniform(-3.4, 3.4, (3, N)))


class Filled:
    """All device memory taken but the last `left` bytes."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        gc.collect()  # contexts that earlier tests left behind
        gc.disable()
        torch.cuda.synchronize()
        self.held = []
        step = 1 << 34
        while step >= 1 << 21:
            free = torch.cuda.mem_get_info()[0]
            if free < self.left + step:
                step >>= 1
                continue
            try:
                self.held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                step >>= 1

    def __exit__(self, *a):
        self.held.clear()
        torch.cuda.empty_cache()
        gc.enable()


def _status(call):
    with pytest.raises(B.BDError) as e:
        call()
    return e.value.status


@pytest.mark.parametrize("precision,block", [("fp64", 1), ("fp32", 1), ("fp32", 4)])
def test_rows_that_cannot_grow(precision, block):
    v = np.random.default_rng(3).normal(size=3 * N)
    c, ref = _context(precision, block), _context(precision, block)
    _condense(ref)
    ref.calc_hi()  # loads every kernel used below
    full = ref.mobility_apply(v)
    ref.close()
    _spread(c)
    c.calc_hi()
    before = c.mobility_apply(v)
    _condense(c)
    with Filled(32 << 20):
        assert _status(c.calc_hi) == OOM
        assert _status(lambda: c.mobility_apply(v)) == STATE
        assert _status(c.calc_hi) == OOM
    c.calc_hi()
    assert np.array_equal(c.mobility_apply(v), full)
    _spread(c)
    c.calc_hi()
    assert np.array_equal(c.mobility_apply(v), before)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_first_build_and_first_solve_without_memory(precision):
    v = np.random.default_rng(4).normal(size=3 * N)
    ref = _context(precision, 4)
    _spread(ref)
    ref.calc_hi()
    want = ref.lanczos_sqrt(v)[0]
    ref.close()
    c = _context(precision, 4)
    _spread(c)
    with Filled(4 << 20):
        assert _status(c.calc_hi) == OOM
        assert _status(lambda: c.mobility_apply(v)) == STATE
        assert _status(c.calc_hi) == OOM
    c.calc_hi()
    with Filled(4 << 20):
        assert _status(lambda: c.lanczos_sqrt(v)) == OOM
        assert _status(lambda: c.lanczos_sqrt(v)) == OOM
    assert np.array_equal(c.lanczos_sqrt(v)[0], want)
