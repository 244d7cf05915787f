"""Neighbour rows built by a warp per bead: caps held in shared memory and the
first one that is not, boxes of fewer than three cells a side and of many, bead
counts that leave a block part empty; the half lists equal the oracle's, entry
by entry, and a row past its cap is an error."""
import numpy as np
import pytest

import bd_b200 as B
import oracle as O

pytestmark = pytest.mark.gpu


def _context(flow, Nb, Nc, L, maxnb):
    x, y, z = B.random_chains(Nb, Nc, L, 3 * Nb + Nc, bond=2.0, min_sep=1.2)
    x, y = B.lab_frame(flow, x, y)
    c = B.Context(B.make_params(flow, Nb, Nc, L, 0.2, 5e-4, max_neighbors=maxnb))
    o = O.Oracle(flow, Nb, Nc, L, 0.2, 5e-4)
    o.lattice(0)
    if flow == 1:
        o.rotate(x, y, 0)
    o.apply_pbc(x, y, z)
    c.set_positions(x, y, z)
    c.set_time(0, 0)
    c.update_lattice(0)
    return c, o, (x, y, z)


@pytest.mark.parametrize("maxnb", [256, 2560, 2561])
@pytest.mark.parametrize("flow,Nb,Nc,L", [(0, 7, 9, 10.0), (1, 7, 9, 13.5), (0, 5, 1, 30.0),
                                          (1, 25, 20, 26.0), (0, 50, 12, 42.0)])
def test_rows_match_oracle(flow, Nb, Nc, L, maxnb):
    c, o, (x, y, z) = _context(flow, Nb, Nc, L, maxnb)
    c.build_neighbors()
    cnt, rows = c.neighbors(256)
    ocnt, orows = o.verlet(x, y, z, 256)
    assert np.array_equal(cnt, ocnt)
    for i in range(Nb * Nc):
        assert np.array_equal(rows[i, :cnt[i]], orows[i, :cnt[i]])


def test_row_past_its_cap_is_an_error():
    c, _, _ = _context(0, 7, 9, 10.0, 8)
    with pytest.raises(B.BDError):
        c.build_neighbors()
        c.sync()
