"""The sequential charge-hop sweep at the edges of its windows of 32 charges
(one charge, one window less, exactly and more than full, several windows),
with most sites taken, so that charges move into sites others have left in the
same and in earlier windows; and with beads at the same position, where single
pair energies are infinite.  Trials, sites and the generator's position agree
exactly with the CPU model of the reference's sweep, which recomputes the whole
energy for every trial."""
import numpy as np
import pytest

import bd_b200 as B
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", [0, 1])
@pytest.mark.parametrize("nch,coincident", [(1, False), (2, False), (31, False), (32, False),
                                            (33, False), (97, False), (140, False), (97, True)])
def test_windows_match_model(flow, nch, coincident):
    Nb, Nc, L = 25, 6, 14.0
    x, y, z = B.random_chains(Nb, Nc, L, 5 + nch, bond=2.0, min_sep=1.6)
    x, y = B.lab_frame(flow, x, y)
    q = np.sort(np.random.default_rng(nch).permutation(Nb * Nc)[:nch]).astype(np.int32)
    q = q[np.random.default_rng(nch + 1).permutation(nch)].copy()
    if coincident:  # empty beads moved onto charged ones
        empty = np.setdiff1d(np.arange(Nb * Nc), q)[:12]
        for e, b in zip(empty, q[::8]):
            x[e], y[e], z[e] = x[b], y[b], z[b]
    kw = dict(barrier=0.1, barrier2=0.2, MStep=1)
    o = O.Oracle(flow, Nb, Nc, L, 0.2, 5e-4, **kw)
    c = B.Context(B.make_params(flow, Nb, Nc, L, 0.2, 5e-4, seed=777, **kw))
    o.lattice(0)
    if flow == 1:
        o.rotate(x, y, 0)
    o.apply_pbc(x, y, z)
    c.set_positions(x, y, z)
    c.set_charges(q)
    track, old = q.copy(), q.copy()
    rng = O.fresh_rng(777)
    moved = 0
    for sweep in range(3):
        o.lattice(sweep)
        _, log = o.charge_hop(x, y, z, track, old, rng)
        c.set_time(sweep)
        c.update_lattice(sweep)
        c.charge_hop()
        assert np.array_equal(c.hop_log(), log), sweep
        tr, od, fl = c.charges()
        assert np.array_equal(tr, track) and np.array_equal(od, old), sweep
        assert fl.sum() == nch and np.all(fl[tr] == 1)
        moved += (log[:, 0] == 1).sum()
    st = c.rng()
    assert (st.idum, st.iy) == (rng.idum, rng.iy)
    assert moved > 0 or nch < 31
