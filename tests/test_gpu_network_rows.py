"""The network's neighbour features from rows of many batches of 32 beads with
equal distances (a cubic lattice, exact coordinates: ties go by index), from
rows shorter than the slots and from empty ones, and its passes at bead counts
around the matrix tiles: the predicted blocks, the loss and the gradient against
oracle/mpnn_oracle.py with the same BF16 operand rounding, to the tolerances
that the pass has on ordinary systems (1e-4; gradients 2e-3)."""
import numpy as np
import pytest

import bd_b200 as B
import mpnn_oracle as Q
import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu


def _check(x, y, z, L, max_neighbors):
    N = len(x)
    o = O.Oracle(0, N, 1, L, 0.2, 5e-4)
    c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                pme_rc=8.0, max_neighbors=max_neighbors))
    o.lattice(0)
    o.apply_pbc(x, y, z)
    c.set_positions(x, y, z)
    c.set_time(0, 0)
    c.update_lattice(0)
    c.build_neighbors()
    r = np.random.default_rng(8)
    w = (B.mpnn_init(7) + r.normal(0, 0.05, B.mpnn_param_count())).astype(np.float32)
    c.mpnn_set_params(w)
    c.mpnn_features()
    cand = [np.setdiff1d(np.nonzero((abs(x - x[i]) < 7) & (abs(y - y[i]) < 7)
                                    & (abs(z - z[i]) < 7))[0], [i]) for i in range(N)]
    nbr, nvec, rbf = Q.features(lambda i, j: o.nid(x, y, z, i, int(j)), cand, N)
    cm = Q.forward(w.astype(np.float64), nbr, nvec, rbf)
    assert rel_err(c.mpnn_predict(), cm["G"]) < 1e-4
    zz, tt = r.normal(size=(N, 3)), r.normal(size=(N, 3)) * 0.5
    loss, grad = c.mpnn_loss_grad(zz.reshape(-1), tt.reshape(-1), want_grad=True)
    lm, gm, _ = Q.loss_grad(w.astype(np.float64), nbr, nvec, rbf, zz, tt)
    assert abs(loss - lm) < 1e-4 * abs(lm)
    at = 0
    for name, shp in Q.LAYOUT:
        n = int(np.prod(shp))
        scale = np.abs(gm[at:at + n]).max()
        assert np.abs(grad[at:at + n] - gm[at:at + n]).max() <= 2e-3 * scale + 1e-12, name
        at += n


@pytest.mark.parametrize("side,alone", [(6, 1), (4, 1), (2, 3), (9, 39), (1, 1)])
def test_lattice_rows_match_model(side, alone):
    L = 60.0
    g = np.stack(np.meshgrid(*[1.5 * np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    far = np.stack([-24.0 + 8.0 * (np.arange(alone) % 6), -24.0 + 8.0 * (np.arange(alone) // 6),
                    np.full(alone, -25.0)], 1)
    pos = np.concatenate([g, far])
    N = len(pos)
    order = np.random.default_rng(side).permutation(N)
    x, y, z = (np.ascontiguousarray(pos[order, d]) for d in range(3))
    _check(x, y, z, L, 1024)


def _clusters(side):
    """side^3 equal clusters of 27 beads, 16 apart, all coordinates exact except
    where a cluster lies across the cell's wall."""
    L = 16.0 * side if side > 1 else 64.0
    a = np.stack(np.meshgrid(*[1.5 * np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    b = np.stack(np.meshgrid(*[16.0 * np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x, y, z = (np.ascontiguousarray(v) for v in (b[:, None] + a[None]).reshape(-1, 3).T)
    N = len(x)
    o = O.Oracle(0, N, 1, L, 0.2, 5e-4)
    o.lattice(0)
    o.apply_pbc(x, y, z)
    c = B.Context(B.make_params(0, N, 1, L, 0.2, 5e-4, mobility="pme", noise="philox",
                                pme_rc=8.0))
    c.set_positions(x, y, z)
    c.set_time(0, 0)
    c.update_lattice(0)
    c.build_neighbors()
    r = np.random.default_rng(8)
    c.mpnn_set_params((B.mpnn_init(7) + r.normal(0, 0.05, B.mpnn_param_count()))
                      .astype(np.float32))
    c.mpnn_features()
    zz, tt = (np.tile(r.normal(size=(27, 3)), (side ** 3, 1)).reshape(-1) for _ in range(2))
    loss, grad = c.mpnn_loss_grad(zz, tt, want_grad=True)
    whole = (np.ptp(np.stack([x, y, z]).reshape(3, -1, 27), axis=2) < 4).all(0)
    return c.mpnn_predict().reshape(-1, 27, 3, 3)[whole], loss, grad


def test_tiles_of_64_rows_match_tiles_of_16():
    """512 equal clusters, more beads than 148 tiles of 64 rows hold, against one
    of them: each row's sums run in the same order in both tiles, so the blocks
    are equal to the last bit; 512 is a power of two, so the loss gradient's
    operands round alike and only the order of its FP32 sums over 13 824 beads
    differs."""
    G1, l1, g1 = _clusters(1)
    G, l, g = _clusters(8)
    assert len(G) >= 343 and np.array_equal(G, np.broadcast_to(G1, G.shape))
    assert abs(l - l1) < 1e-5 * abs(l1)
    at = 0
    for name, shp in Q.LAYOUT:
        n = int(np.prod(shp))
        scale = np.abs(g1[at:at + n]).max()
        assert np.abs(g[at:at + n] - g1[at:at + n]).max() <= 2e-3 * scale, name
        at += n
