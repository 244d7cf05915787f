"""Parallel charge-hop sweep with few, full cells: one cell for the whole box
and two per direction, so that a cell's trials span several groups of 32 and
charges move into sites that others left in the same colour.  Against
oracle/hop_oracle.py: decisions, sites and flags agree exactly; Ewald energies
to the particle mesh's accuracy (1e-5 kT, as on small cells)."""
import numpy as np
import pytest

import bd_b200 as B
import hop_oracle as H
import oracle as O
import pme_oracle as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [14.0, 40.0])
@pytest.mark.parametrize("coulomb", ["dh", "ewald"])
@pytest.mark.parametrize("flow", [0, 1])
def test_full_cells_match_model(flow, coulomb, radius):
    Nb, Nc, L, seed = 25, 14, 30.0, 11 + flow
    x, y, z = B.random_chains(Nb, Nc, L, seed, bond=2.0, min_sep=2.0)
    x, y = B.lab_frame(flow, x, y)
    track = B.random_charges(Nb, Nc, 0.6, seed + 1)
    qk = np.where((track // Nb) % 2 == 0, 1.0, -1.0)
    c = B.Context(B.make_params(flow, Nb, Nc, L, 0.2, 5e-4, noise="philox", hop="parallel",
                                coulomb=coulomb, hop_radius=radius, philox_seed=300 + seed,
                                Ncharges=len(track), barrier=0.05, barrier2=0.1))
    c.set_positions(x, y, z)
    c.set_charges(track)
    c.set_charge_values(qk)
    c.set_time(0, 0)
    c.update_lattice(0)
    c.transform_coords()
    c.apply_pbc()
    c.build_neighbors()
    px, py, pz = (np.array(a) for a in c.positions())
    _, _, flags0 = c.charges()
    c.charge_hop()
    tr, _, fl = c.charges()
    log, de = c.hop_log(), c.hop_energies()
    o = O.Oracle(flow, Nb, Nc, L, 0.2, 5e-4)
    o.lattice(0)
    s = o.s
    Hc = P.reduced_cell(list(s.L1), list(s.L2), L)
    cth, sth = (s.cth, s.sth) if flow == 1 else (1.0, 0.0)
    rc = min(10.0, 0.43 * L)
    ew = H.EwaldTerms(Hc, 3.5 / rc, rc, 2.0) if coulomb == "ewald" else None
    got = H.parallel_sweep(o, px, py, pz, track, qk, flags0, Hc, cth, sth, radius, 2.0, 1 / 5.0,
                           0.05, 0.1, 300 + seed, 0, ewald=ew)
    assert np.array_equal(log, got[2])
    assert np.array_equal(tr, got[0])
    assert np.array_equal(fl, got[3])
    assert np.array_equal(np.isnan(de), log[:, 0] == 0)
    # several moves, one of them into a site that was occupied when the sweep began
    accepted = log[:, 0] == 1
    assert accepted.sum() > 20
    assert np.isin(log[accepted, 1], track).any()
    if ew is not None:
        ev = ~np.isnan(got[4])
        assert np.abs(de[ev] - got[4][ev]).max() < 1e-5
