"""The two forms of the real-space rows (whole FP32 tensors for noise blocks;
t1 and t2 / r^2 with FP64 displacements, inputs and sums otherwise), on both
sides of the rules that give a group of four beads one, two or four warps, and
five packed pairs at each of them, against oracle/pme_oracle.py (FP64 1e-11, FP32
2e-6: weights, grids, transforms and tensors hold 24 bits, 6e-8 each, a result
adds some tens of such roundings)."""
import functools

import numpy as np
import pytest

import bd_b200 as B
import oracle as O
import pme_oracle as P
from conftest import rel_err

pytestmark = pytest.mark.gpu

K, ORDER, RC, ALPHA, T = 32, 4, 6.0, 0.45, 2000
FACTORS = np.array([1.0, -2.0, 3.0, 0.5, -1.25, 0.75, 2.5, -0.375, 1.5])


@functools.lru_cache(maxsize=None)
def _system(N):
    """Positions, the cell of a sheared step, a vector and its product."""
    L = max(24.0, (N / 0.02) ** (1 / 3))
    r = np.random.default_rng(N)
    x, y, z = (np.ascontiguousarray(v) for v in r.uniform(-L / 2, L / 2, (3, N)))
    o = O.Oracle(0, N, 1, L, 0.2, 5e-4)
    o.lattice(T)
    o.apply_pbc(x, y, z)
    H = P.reduced_cell(list(o.s.L1), list(o.s.L2), L)
    v = r.normal(size=(N, 3))
    ref = P.pme_apply(H, np.stack([x, y, z], 1), v, K, ORDER, ALPHA, RC,
                      alpha_ref=P.ref_alpha(T, o.s.tp, o.s.L2yp))
    return L, (x, y, z), v.reshape(-1), ref.reshape(-1)


FORMS = pytest.mark.parametrize("precision,block", [("fp64", 1), ("fp64", 9), ("fp32", 1),
                                                    ("fp32", 9)])


def _check(N, Nb, precision, block):
    L, pos, v, ref = _system(N)
    c = B.Context(B.make_params(0, Nb, N // Nb, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision=precision, pme_grid=K, pme_order=ORDER, pme_rc=RC,
                                pme_alpha=ALPHA, noise_block=block))
    c.set_positions(*pos)
    c.set_time(T, T)
    c.update_lattice(T)
    c.calc_hi()
    tol = 1e-11 if precision == "fp64" else 2e-6
    assert rel_err(c.mobility_apply(v), ref) < tol
    for k in (2, 4, 5, 8, 9) if block > 1 else ():  # an odd last vector among them
        got = c.mobility_apply_block(FACTORS[:k, None] * v)
        assert max(rel_err(got[r], FACTORS[r] * ref) for r in range(k)) < tol, k


@FORMS
@pytest.mark.parametrize("N", [2, 33, 2364, 2365, 7104, 7105, 9469, 14205, 23677])
def test_forms_match_model(N, precision, block):
    _check(N, N, precision, block)


@FORMS
@pytest.mark.parametrize("N,Nb", [(2, 1), (33, 11), (33, 3), (7105, 1), (7105, 7), (7105, 5),
                                  (7104, 2)])
def test_beads_grouped_in_space_match_model(N, Nb, precision, block):
    """Short chains, whose groups follow the space and not the index."""
    _check(N, Nb, precision, block)


@pytest.mark.parametrize("precision,block", [("fp64", 1), ("fp32", 4)])
def test_monomers_need_no_longer_rows(precision, block):
    """Beads in no spatial order: grouped by index, four of them would share hardly
    a neighbour and their rows overflow the default cap."""
    N, L = 8000, 60.0
    r, used = np.random.default_rng(9), {}
    chains = np.stack(B.random_chains(100, N // 100, L, 3), 1)
    for Nb, pos in ((100, chains), (1, r.uniform(-L / 2, L / 2, (N, 3)))):
        c = B.Context(B.make_params(0, Nb, N // Nb, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                    precision=precision, noise_block=block, pme_rc=12.1))
        c.set_positions(*(np.ascontiguousarray(a) for a in pos.T))
        c.set_time(0, 0)
        c.update_lattice(0)
        c.apply_pbc()
        c.calc_hi()
        used[Nb] = c.device_bytes()
        c.close()
    assert used[1] < 1.1 * used[100], used


def test_single_vector_contexts_take_fp64_inputs():
    """FP32 storage with one right-hand side: an input that differs by less than
    FP32 resolves reaches the neighbours through the real-space tensors (the mesh
    takes FP32 values and does not see it).  The tensors hold 24 bits (1e-7 of
    values below one), the difference of two FP64 results 2^-30 apart some units
    of 2^-53 2^30 = 1.2e-7."""
    N, L, rc, alpha, j, h = 300, 24.0, 9.0, 0.4, 7, 2.0 ** -30
    pos = np.random.default_rng(8).uniform(-L / 2, L / 2, (N, 3))
    c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                precision="fp32", pme_rc=rc, pme_alpha=alpha))
    c.set_positions(*(np.ascontiguousarray(a) for a in pos.T))
    c.set_time(0, 0)
    c.update_lattice(0)
    c.calc_hi()
    d = pos - pos[j]
    d -= L * np.rint(d / L)
    rr = (d * d).sum(1)
    pairs = np.flatnonzero((rr >= 4.0) & (rr < rc * rc))
    t1, t2 = P.real_terms(alpha, rr[pairs])
    for a in range(3):
        v = np.zeros((N, 3))
        v[j, a] = 1.0
        low = c.mobility_apply(v.reshape(-1)).reshape(N, 3)
        v[j, a] += h
        step = (c.mobility_apply(v.reshape(-1)).reshape(N, 3) - low) / h
        want = (t2 / rr[pairs] * d[pairs, a])[:, None] * d[pairs]
        want[:, a] += t1
        assert np.abs(step[pairs] - want).max() < 1e-6
        far = np.flatnonzero(rr > rc * rc)
        assert np.abs(step[far]).max() == 0.0


@pytest.mark.parametrize("precision,block,most", [("fp64", 1, 20), ("fp64", 4, 20), ("fp32", 1, 12),
                                                  ("fp32", 4, 28)])
def test_memory_of_an_explicit_pair_cap(precision, block, most):
    """An entry of the cap costs a bead at most an index and its own pair's
    numbers (FP64 4 + 16 bytes; FP32 4 + 8, with blocks 4 + 8 + 16)."""
    N, L = 10000, 82.0  # four beads' caps stay below N
    pos = np.random.default_rng(5).uniform(-L / 2, L / 2, (3, N))
    used = []
    for cap in (1024, 2048):
        c = B.Context(B.make_params(0, 50, N // 50, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                    precision=precision, noise_block=block, pme_rc=10.0,
                                    pme_max_pairs=cap))
        c.set_positions(*pos)
        c.set_time(0, 0)
        c.update_lattice(0)
        c.calc_hi()
        used.append(c.device_bytes())
        c.close()
    assert used[1] - used[0] <= most * N * 1024


def test_explicit_cap_grows_rows_of_four_beads():
    """Rows start with the cap of one bead: four beads whose neighbourhoods differ
    need more, up to four times as much, and no bead's pairs are lost."""
    N, L = 2000, 40.0
    r = np.random.default_rng(6)
    pos, v = r.uniform(-L / 2, L / 2, (3, N)), r.normal(size=3 * N)
    out = []
    for cap in (0, 200):  # mean 131 pairs a bead, in no spatial order
        c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                    precision="fp64", pme_rc=10.0, pme_max_pairs=cap))
        c.set_positions(*pos)
        c.set_time(0, 0)
        c.update_lattice(0)
        c.calc_hi()
        out.append(c.mobility_apply(v))
    assert np.array_equal(out[0], out[1])


def _compact(Nb, Nc, spacing):
    """Chains folded on a cubic lattice, consecutive beads on neighbouring sites."""
    N = Nb * Nc
    m = int(np.ceil(N ** (1 / 3)))
    i = np.arange(N)
    z, y, x = i // (m * m), i // m % m, i % m
    y = np.where(z % 2, m - 1 - y, y)
    x = np.where((i // m) % 2, m - 1 - x, x)
    return [(a - (m - 1) / 2) * spacing for a in (x, y, z)]


@pytest.mark.parametrize("precision,block", [("fp64", 1), ("fp32", 1), ("fp32", 4)])
def test_rows_grow_between_the_steps_of_a_run(precision, block):
    """A run whose chains have collapsed by the next mobility build: the rows grow,
    and the captured iterations of the earlier steps are not used on them.  The
    steps equal those of a run that starts there, but for where the Krylov runs
    stop (tolerance 1e-6)."""
    Nb, Nc, L = 50, 80, 60.0

    def run():
        c = B.Context(B.make_params(0, Nb, Nc, L, 0.01, 5e-4, mobility="pme", noise="philox",
                                    precision=precision, noise_block=block, pme_rc=12.0,
                                    philox_seed=3))
        c.set_time(0, 0)
        c.update_lattice(0)
        return c

    compact = _compact(Nb, Nc, 2.05)
    moved = []
    for collapsed in (False, True):
        c = run()
        if not collapsed:
            c.set_positions(*B.random_chains(Nb, Nc, L, 4, bond=2.0, min_sep=1.9))
            c.step_lanczos(0, 4, with_hop=False)
            small = c.device_bytes()
        else:
            for _ in range(4):  # the draws of the other run's first steps
                c.get_noise()
        c.noise_block_release()
        c.set_positions(*compact)
        c.build_neighbors()  # positions set from outside: the lists are not told
        c.step_lanczos(100, 4, with_hop=False)
        moved.append(np.stack(c.positions()) - np.stack(compact))
        if not collapsed:
            assert c.device_bytes() > small  # the rows did grow
        c.close()
    assert rel_err(moved[0], moved[1]) < 1e-5
