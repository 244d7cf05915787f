"""FP32 contexts hold the spline weights in FP64: a bead that moves by less than FP32
weights resolve sees the interpolated field change.  The bead has no input of its
own, so the grid does not change, and no neighbour within the cutoff.  The change of
its output over a millionth of a grid spacing along y and z agrees with the FP64
context's to 1e-3: the grid's values differ by some 1e-7 of the field's size, their
differences over a spacing by as much of a few times their own, and FP64 sums over
the stencil add 1e-16 / 1e-6; FP32 weights (6e-8 of 1e-6) would leave a tenth.
(Along x the sums over the stencil's levels are FP32.)"""
import numpy as np
import pytest

import bd_b200 as B

pytestmark = pytest.mark.gpu

N, L, K, RC = 300, 30.0, 40, 5.0


def _output(precision, block, pos, v):
    c = B.Context(B.make_params(0, 20, N // 20, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_rc=RC, pme_alpha=0.6,
                                noise_block=block))
    c.set_positions(*(np.ascontiguousarray(a) for a in pos.T))
    c.set_time(0, 0)
    c.update_lattice(0)
    c.calc_hi()
    out = [c.mobility_apply(v)]
    if block > 1:
        out.append(c.mobility_apply_block(np.stack([v, -v, 2 * v])[:block])[0])
    c.close()
    return [o.reshape(N, 3)[0] for o in out]


@pytest.mark.parametrize("axis", [1, 2])
def test_weights_resolve_small_moves(axis):
    r = np.random.default_rng(12)
    pos = np.empty((N, 3))
    pos[0] = (0.31, -0.17, 0.23)
    n = 1
    while n < N:  # the others keep out of the first one's cutoff
        p = r.uniform(-L / 2, L / 2, 3)
        if np.linalg.norm(p - pos[0]) > RC + 0.5:
            pos[n] = p
            n += 1
    v = r.normal(size=(N, 3))
    v[0] = 0.0
    v = v.reshape(-1)
    moved = pos.copy()
    moved[0, axis] += 1e-6 * L / K
    want = _output("fp64", 1, moved, v)[0] - _output("fp64", 1, pos, v)[0]
    for block in (1, 3):
        for a, b in zip(_output("fp32", block, moved, v), _output("fp32", block, pos, v)):
            assert np.linalg.norm(a - b - want) < 1e-3 * np.linalg.norm(want)
