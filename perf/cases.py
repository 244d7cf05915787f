"""Performance cases: the work a Brownian-dynamics program has this library do.

Every case goes through the public binding (``bd_b200.Context``), whose calls
take and return host arrays as the C ABI does: positions, noise vectors and
charges go in, positions, forces, displacements and charge tracks come out.
Systems are seeded chains at the bead density of the 8000-bead workload
(box edge 60), alternately poly-anionic and poly-cationic.  Contexts with
FP32 storage return FP32 arrays here: that is the precision their products
are held in.

``exact`` evaluates the same operators in FP64 with plain torch: the
particle-mesh mobility on the same grid, its square root by
eigen-decomposition, the pair and Ewald forces, and the network's gradient.
Whole Brownian steps have no such value (their noise is the library's own
generator, their displacement an iterative solve).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "smdlt-ca-chrg-flow_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import bd_b200 as B  # noqa: E402

DENSITY = 8000 / 60.0 ** 3
CUTOFFS = (0.0,) + tuple(B.PME_CUTOFFS)  # 0: the default cutoff, 10 or 0.43 of the box


def _steps(name, **kw):
    return dict(dict(kind="steps", name=name, flow=1, Nb=100, Nc=80, wi=2.0, precision="fp32",
                     precond="learned", rc=0.0, block=10, steps=10), **kw)


def listed():
    return [
        # the reference's own small shear case (500 beads): launch-bound steps
        _steps("steps_500_shear", flow=0, Nb=25, Nc=20, wi=1.0, precond="segment"),
        # a dilute extensional run of 8000 beads, cutoff as autotuned
        _steps("steps_8k_ext", rc=12.1),
        # the 50 000-bead extensional run that the headline is quoted on
        _steps("steps_50k_ext", Nc=500, wi=3.0, rc=14.5),
        # the largest: a semidilute solution of 200 000 beads in shear
        _steps("steps_200k_shear", flow=0, Nc=2000, wi=10.0, rc=15.5),
        # the plain FP64 method, chosen where FP32 products are not wanted
        _steps("steps_8k_fp64", precision="fp64", precond="none", rc=12.1),
        # the mobility product of several vectors, for a caller's own solver
        # (an odd number of right-hand sides, chains of 25: ragged sizes)
        dict(kind="product", name="product_7_vectors", flow=0, Nb=25, Nc=331, precision="fp32",
             rc=0.0, k=7),
        # the periodic mobility rebuild with one product after it
        dict(kind="rebuild", name="rebuild_50k", flow=1, Nb=100, Nc=500, precision="fp32",
             rc=14.5, k=10),
        # one Brownian displacement per call, FP64, no preconditioner (the
        # library's defaults)
        dict(kind="sqrt", name="sqrt_1k_fp64", flow=1, Nb=50, Nc=20, precision="fp64", rc=0.0),
        # bond, excluded-volume and Ewald Coulomb forces of one step
        dict(kind="forces", name="forces_50k", flow=1, Nb=100, Nc=500, rc=14.5),
        # one charge-hop sweep with Ewald energies
        dict(kind="hop", name="hop_50k", flow=1, Nb=100, Nc=500, rc=14.5),
        # the reference's own algorithm: dense hybrid mobility, CA-TEA,
        # Debye-Hueckel, sequential charge hops every 5 steps
        dict(kind="reference", name="reference_500", flow=0, Nb=25, Nc=20, steps=10),
        # forward and backward pass of the preconditioner network
        dict(kind="network", name="network_2k", flow=0, Nb=50, Nc=40),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _chains(rng, lo, hi, lengths=(25, 50, 75, 100)):
    Nb = rng.choice(lengths)
    return Nb, max(2, round(_log(rng, lo, hi) / Nb))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "product", "rebuild", "sqrt",
                       "forces", "hop", "reference", "network"])
    c = dict(kind=kind, flow=rng.randrange(2))
    if kind == "steps":
        c["precision"] = rng.choice(["fp32", "fp32", "fp64"])
        hi = 100000 if c["precision"] == "fp32" else 12000
        c["Nb"], c["Nc"] = _chains(rng, 500, hi)
        c["wi"] = rng.uniform(0.5, 10.0)
        c["precond"] = rng.choice(["none", "segment", "learned"])
        c["rc"] = rng.choice(CUTOFFS)
        c["block"] = rng.randrange(2, 11)
        c["steps"] = c["block"]
    elif kind == "product":
        c["precision"] = rng.choice(["fp32", "fp64"])
        c["Nb"], c["Nc"] = _chains(rng, 500, 20000)
        c["rc"], c["k"] = rng.choice(CUTOFFS), rng.randrange(1, 11)
    elif kind == "rebuild":
        c["precision"] = rng.choice(["fp32", "fp64"])
        c["Nb"], c["Nc"] = _chains(rng, 1000, 50000)
        c["rc"], c["k"] = rng.choice(CUTOFFS), rng.randrange(1, 11)
    elif kind == "sqrt":
        c["precision"] = rng.choice(["fp32", "fp64"])
        c["Nb"], c["Nc"] = _chains(rng, 500, 1200, (25, 50))
        c["rc"] = 0.0
    elif kind in ("forces", "hop"):
        c["Nb"], c["Nc"] = _chains(rng, 1000, 50000)
        c["rc"] = rng.choice(CUTOFFS)
    elif kind == "reference":
        c["Nb"], c["Nc"] = _chains(rng, 300, 1000, (25, 50))
        c["steps"] = rng.randrange(3, 11)
    else:
        c["Nb"], c["Nc"] = _chains(rng, 500, 8000, (25, 50, 100))
    return c


# ---------------------------------------------------------------------------
# systems


def _box(c):
    return (c["Nb"] * c["Nc"] / DENSITY) ** (1.0 / 3.0)


def _cutoff(c):
    """The context's cutoff parameter: at most the minimum-image bound."""
    rc = c.get("rc", 0.0)
    return min(rc, 0.43 * _box(c)) if rc > 0 else 0.0


def _walks(Nb, Nc, L, r):
    """Self-avoiding chains on a jittered cubic lattice of spacing 2 or a
    little more, all chains grown together (a chain that gets stuck starts
    again): N x 3 positions, nearest beads at least 1.8 apart."""
    m = int(L // 2.0)
    used = np.zeros(m ** 3, bool)
    steps = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]])
    site = -np.ones((Nc, Nb), np.int64)
    todo = np.arange(Nc)

    def flat(q):
        return (q[..., 0] * m + q[..., 1]) * m + q[..., 2]

    while len(todo):
        free = np.flatnonzero(~used)
        head = r.choice(free, len(todo), replace=False)
        used[head] = True
        site[todo, 0] = head
        live = todo
        for b in range(1, Nb):
            grown = np.zeros(len(live), bool)
            for _ in range(12):
                w = np.flatnonzero(~grown)
                if not len(w):
                    break
                h = site[live[w], b - 1]
                q = np.stack([h // (m * m), (h // m) % m, h % m], 1)
                nxt = flat((q + steps[r.integers(0, 6, len(w))]) % m)
                ok = ~used[nxt]
                w, nxt = w[ok], nxt[ok]
                nxt, first = np.unique(nxt, return_index=True)
                w = w[first]
                used[nxt] = True
                site[live[w], b] = nxt
                grown[w] = True
            stuck = live[~grown]
            if len(stuck):
                s = site[stuck, :b]
                used[s.reshape(-1)] = False
                site[stuck] = -1
                live = live[grown]
        todo = np.flatnonzero((site < 0).any(1))
    s = site.reshape(-1)
    q = np.stack([s // (m * m), (s // m) % m, s % m], 1)
    x = (q + 0.5) * (L / m) - L / 2 + r.uniform(-0.1, 0.1, (len(s), 3))
    # one random shift of the whole system, wrapped back into the box
    x += r.uniform(-L / 2, L / 2, 3)
    return x - L * np.round(x / L)


def _system(c, seed):
    r = np.random.default_rng([seed, c["Nb"], c["Nc"]])
    p = _walks(c["Nb"], c["Nc"], _box(c), r)
    x, y = B.lab_frame(c["flow"], p[:, 0], p[:, 1])
    x, y, z = (np.ascontiguousarray(a) for a in (x, y, p[:, 2]))
    k = c["Nb"] // 2
    q = np.argsort(r.random((c["Nc"], c["Nb"])), 1)[:, :k] + np.arange(c["Nc"])[:, None] * c["Nb"]
    q = np.sort(q, 1).reshape(-1).astype(np.int32)
    qk = np.where((q // c["Nb"]) % 2 == 0, -1.0, 1.0)
    return x, y, z, q, qk, r


def _tau(Nb):
    return 175.0 * (Nb / 50.0) ** (3 * 0.588)


def _context(c, seed, **extra):
    """A particle-mesh context on the seeded system, in the frame the force
    and mobility routines read (bead positions wrapped, rotated in extension)."""
    x, y, z, q, qk, r = _system(c, seed)
    kw = dict(Ncharges=len(q), shear_kappas_override=1, noise="philox", philox_seed=seed + 1,
              mobility="pme", precision=c.get("precision", "fp32"), coulomb="ewald",
              hop="parallel", pme_rc=_cutoff(c), lanczos_max=200)
    kw.update(extra)
    ctx = B.Context(B.make_params(c["flow"], c["Nb"], c["Nc"], _box(c),
                                  c.get("wi", 2.0) / _tau(c["Nb"]), 5e-4, **kw))
    ctx.set_positions(x, y, z)
    ctx.set_charges(q)
    ctx.set_charge_values(qk)
    ctx.set_time(0, 0)
    ctx.update_lattice(0)
    ctx.transform_coords()
    ctx.apply_pbc()
    ctx.build_neighbors()
    return ctx, q, qk, r


def _precondition(ctx, c):
    kind = c["precond"]
    if kind == "none":
        return
    if kind == "learned":
        ctx.mpnn_set_params(np.load(os.path.join(PKG, "mpnn_params.npy")))
    ctx.set_preconditioner(kind, 10 if c["Nb"] % 10 == 0 else 5)


def _held(c, a):
    return np.asarray(a, np.float32) if c.get("precision") == "fp32" else np.asarray(a)


def prepare(case, seed):
    c = dict(case)
    s = dict(case=c)
    kind = c["kind"]
    if kind == "steps":
        ctx, _, _, _ = _context(c, seed, noise_block=c["block"])
        _precondition(ctx, c)
        ctx.inverse_coords()
        # the first step builds the mobility that later steps use
        ctx.step_lanczos(0, 1, with_hop=False)
        ctx.noise_block_release()
        s.update(ctx=ctx, at=ctx.positions())
    elif kind == "product":
        ctx, _, _, r = _context(c, seed, noise_block=c["k"])
        ctx.calc_hi()
        s.update(ctx=ctx, V=r.normal(size=(c["k"], 3 * ctx.N)))
    elif kind == "rebuild":
        ctx, _, _, r = _context(c, seed, noise_block=c["k"])
        s.update(ctx=ctx, V=r.normal(size=3 * ctx.N))
    elif kind == "sqrt":
        ctx, _, _, r = _context(c, seed)
        ctx.calc_hi()
        s.update(ctx=ctx, V=r.normal(size=3 * ctx.N))
    elif kind == "forces":
        s.update(ctx=_context(c, seed)[0])
    elif kind == "hop":
        ctx, q, qk, _ = _context(c, seed)
        s.update(ctx=ctx, q=q, qk=qk)
    elif kind == "reference":
        x, y, z, q, _, r = _system(c, seed)
        p = B.make_params(c["flow"], c["Nb"], c["Nc"], _box(c), 1.0 / _tau(c["Nb"]), 5e-4,
                          Ncharges=len(q), MStep=5, spring="Hookean", kappas=200.0, qmax=2.0,
                          epsilon=0.1, seed=-(seed % 100000) - 1)
        ctx = B.Context(p)
        ctx.build_grid(0.001)
        for sb in range(21):
            ctx.set_tea(sb, r.uniform(0.3, 0.6), r.uniform(0.8, 1.0, 3 * c["Nb"]))
        ctx.set_positions(x, y, z)
        ctx.set_charges(q)
        ctx.set_time(0, 0)
        ctx.update_lattice(0)
        ctx.step_reference(0, 1, False)
        s.update(ctx=ctx, at=ctx.positions(), q=q, rng=ctx.rng())
    else:
        ctx, _, _, r = _context(c, seed)
        w = B.mpnn_init(seed) + r.normal(0, 0.05, B.mpnn_param_count()).astype(np.float32)
        z = r.normal(size=3 * ctx.N)
        s.update(ctx=ctx, w=w, z=z, t=z + 0.3 * r.normal(size=3 * ctx.N))
    return s


def run(s):
    c, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "steps":
        ctx.set_positions(*s["at"])
        ctx.step_lanczos(1, c["steps"], with_hop=False)
        return _held(c, ctx.positions())
    if kind == "product":
        return _held(c, ctx.mobility_apply_block(s["V"]))
    if kind == "rebuild":
        ctx.calc_hi()
        return _held(c, ctx.mobility_apply(s["V"]))
    if kind == "sqrt":
        return _held(c, ctx.lanczos_sqrt(s["V"])[0])
    if kind == "forces":
        ctx.reset_force()
        ctx.bond_force()
        ctx.ev_force()
        ctx.coulomb_force()
        return dict(forces=ctx.forces(), energy=ctx.coulomb_energy()["total"])
    if kind == "hop":
        ctx.set_charges(s["q"])
        ctx.set_charge_values(s["qk"])
        ctx.charge_hop()
        return dict(track=ctx.charges()[0], energy=ctx.hop_energies())
    if kind == "reference":
        ctx.set_positions(*s["at"])
        ctx.set_charges(s["q"])
        ctx.set_rng(s["rng"])
        ctx.step_reference(1, c["steps"], True)
        return dict(positions=np.stack(ctx.positions()), track=ctx.charges()[0])
    ctx.mpnn_set_params(s["w"])
    ctx.mpnn_features()
    loss, grad = ctx.mpnn_loss_grad(s["z"], s["t"], want_grad=True)
    return dict(loss=np.float32(loss), grad=grad)


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _product_flops(c, k):
    """Pairs within the cutoff (18 operations a right-hand side), spreading
    and interpolation (2 x 6 operations a stencil point), transforms."""
    N, L = c["Nb"] * c["Nc"], _box(c)
    rc = _cutoff(c) or min(10.0, 0.43 * L)
    K = B.pme_default_grid(L, rc)
    pairs = 4.0 / 3.0 * math.pi * rc ** 3 * DENSITY * N
    return k * (18.0 * pairs + 12.0 * 512 * N + 3 * 2 * 2.5 * K ** 3 * math.log2(K ** 3))


def work(case):
    c = dict(case)
    N, kind = c["Nb"] * c["Nc"], c["kind"]
    io = 48.0 * N
    if kind == "steps":
        iters = 25.0 * math.log10(N) - 40.0  # Krylov dimension at tolerance 1e-6, about
        iters *= 1.0 if c["precond"] != "none" else 1.25
        return dict(bytes=io, flops=c["steps"] * (iters + 1) * _product_flops(c, 1))
    if kind == "product":
        return dict(bytes=c["k"] * io, flops=_product_flops(c, c["k"]))
    if kind == "rebuild":
        return dict(bytes=io + 24.0 * N, flops=3.0 * _product_flops(c, 1))
    if kind == "sqrt":
        return dict(bytes=io, flops=50 * _product_flops(c, 1))
    if kind == "forces":
        return dict(bytes=io, flops=_product_flops(c, 1))
    if kind == "hop":
        # per trial: the charges within the cutoff of both sites, and the mesh
        # potential once per colour
        return dict(bytes=24.0 * N, flops=N / 2 * (2 * 60 * 80.0 + 2 * 512 * 4)
                    + 8 * _product_flops(c, 1) / 3)
    if kind == "reference":
        return dict(bytes=c["steps"] * 24.0 * N * N, flops=c["steps"] * 2 * 9.0 * N * N)
    edges = 12.0 * N
    return dict(bytes=48.0 * N + 8.0 * 13634, flops=3 * 2 * (edges * 1024 + N * (4096 + 8192)))


# ---------------------------------------------------------------------------
# the same in FP64, plain torch


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spline(f, p):
    """M_p(f + k), k = 0..p-1."""
    a = torch.stack([f, 1.0 - f], -1)
    for n in range(3, p + 1):
        z = torch.zeros_like(f)[:, None]
        hi, lo = torch.cat([a, z], -1), torch.cat([z, a], -1)
        k = torch.arange(n, device=f.device, dtype=f.dtype)
        a = ((f[:, None] + k) * hi + (n - f[:, None] - k) * lo) / (n - 1)
    return a


class _Mesh:
    """Smooth particle-mesh sums on the cubic (in extension rotated) cell."""

    def __init__(self, c, x, y, z, p=8):
        d = _dev()
        self.L, self.p = _box(c), p
        self.rc = _cutoff(c) or min(10.0, 0.43 * self.L)
        self.K = B.pme_default_grid(self.L, self.rc)
        self.r = torch.tensor(np.stack([x, y, z], 1), dtype=torch.float64, device=d)
        L = self.L
        ex, ey = (np.array(B.lab_frame(c["flow"], np.array([L, 0.0]), np.array([0.0, L])))).T
        H = np.array([[ex[0], ey[0], 0.0], [ex[1], ey[1], 0.0], [0.0, 0.0, L]])
        self.H = torch.tensor(H, device=d)
        self.Hi = torch.linalg.inv(self.H)
        s = self.r @ self.Hi.T
        u = (s - torch.floor(s)) * self.K
        b = torch.floor(u)
        f = u - b
        g = (b.long()[:, :, None] - torch.arange(p, device=d)) % self.K
        self.idx = g
        self.w = torch.stack([_spline(f[:, a], p) for a in range(3)], 1)
        lo = torch.stack([_spline(f[:, a], p - 1) for a in range(3)], 1)
        z = torch.zeros_like(lo[..., :1])
        self.dw = torch.cat([lo, z], -1) - torch.cat([z, lo], -1)

    def _chunks(self):
        for i in range(0, len(self.r), 8192):
            s = slice(i, i + 8192)
            g = self.idx[s]
            flat = ((g[:, 0, :, None, None] * self.K + g[:, 1, None, :, None]) * self.K
                    + g[:, 2, None, None, :])
            yield s, flat

    def _w3(self, s, a=None):
        w = [self.dw[s, d] if d == a else self.w[s, d] for d in range(3)]
        return w[0][:, :, None, None] * w[1][:, None, :, None] * w[2][:, None, None, :]

    def spread(self, q):
        Q = torch.zeros(self.K ** 3, dtype=torch.float64, device=q.device)
        for s, flat in self._chunks():
            Q.index_add_(0, flat.reshape(-1), (self._w3(s) * q[s, None, None, None]).reshape(-1))
        return Q.reshape(self.K, self.K, self.K)

    def gather(self, phi, a=None):
        out = torch.zeros(len(self.r), dtype=torch.float64, device=phi.device)
        for s, flat in self._chunks():
            out[s] = (self._w3(s, a) * phi.reshape(-1)[flat]).sum((1, 2, 3))
        return out

    def waves(self):
        K, d = self.K, self.r.device
        m = torch.fft.fftfreq(K, 1.0 / K, device=d, dtype=torch.float64)
        mz = torch.arange(K // 2 + 1, device=d, dtype=torch.float64)
        B3 = 2 * math.pi * self.Hi
        k = (m[:, None, None, None] * B3[0] + m[None, :, None, None] * B3[1]
             + mz[None, None, :, None] * B3[2])
        kk = (k * k).sum(-1)
        M = _spline(torch.zeros(1, device=d, dtype=torch.float64), self.p)[0]
        j = torch.arange(self.p - 1, device=d, dtype=torch.float64)
        e = torch.exp(2j * math.pi * torch.arange(K, device=d)[:, None] * j / K)
        b = 1.0 / (e @ M[1:].to(e.dtype)).abs().square()
        bz = b[: K // 2 + 1]
        return k, kk, b[:, None, None] * b[None, :, None] * bz[None, None, :]

    def near(self, rc, heavy):
        """heavy(i, j, d, rr) for the ordered pairs closer than rc, in pieces."""
        N = len(self.r)
        step = max(1, int(2e7 // N))
        for i0 in range(0, N, step):
            d = self.r[i0:i0 + step, None, :] - self.r[None, :, :]
            s = d @ self.Hi.T
            d = (s - torch.round(s)) @ self.H.T
            rr = (d * d).sum(-1)
            i, j = torch.nonzero(rr < rc * rc, as_tuple=True)
            keep = j != i + i0
            i, j = i[keep], j[keep]
            heavy(i + i0, j, d[i, j], rr[i, j])


def _rpy_real(a, rr, far):
    r = rr.sqrt()
    C1, C3 = 0.75 / r + 0.5 / (r * rr), 0.75 / r - 1.5 / (r * rr)
    C2 = 4 * a ** 7 * rr * rr + 3 * a ** 3 * rr - 20 * a ** 5 * rr - 4.5 * a + 14 * a ** 3 + a / rr
    C4 = (-4 * a ** 7 * rr * rr - 3 * a ** 3 * rr + 16 * a ** 5 * rr + 1.5 * a - 2 * a ** 3
          - 3 * a / rr)
    if not far:
        n = r <= 2.0
        C1, C3 = torch.where(n, 1.0 - 0.28125 * r, C1), torch.where(n, 0.09375 * r, C3)
        C2 = torch.where(n, 64 * a ** 7 + 12 * a ** 3 - 80 * a ** 5 - 4.5 * a + 14 * a ** 3
                         + 0.25 * a + 0 * r, C2)
        C4 = torch.where(n, -64 * a ** 7 - 12 * a ** 3 + 64 * a ** 5 + 1.5 * a - 2 * a ** 3
                         - 0.75 * a + 0 * r, C4)
    ec, ex = torch.erfc(a * r), torch.exp(-a * a * rr) / math.sqrt(math.pi)
    return C1 * ec + C2 * ex, C3 * ec + C4 * ex


class _Mobility(_Mesh):
    """M v of the particle-mesh mobility at time 0 (split 4 / cutoff; calcHI's
    own split 4 / L for overlapping beads)."""

    def __init__(self, c, x, y, z):
        super().__init__(c, x, y, z)
        a = self.a = 4.0 / self.rc
        k, kk, b = self.waves()
        k1 = torch.where(kk > 0, kk, torch.ones_like(kk))
        V = self.L ** 3
        f = ((1 - k1 / 3) * (1 + k1 / (4 * a * a) + k1 * k1 / (8 * a ** 4)) * 6 * math.pi / k1
             * torch.exp(-k1 / (4 * a * a)) / V * b)
        self.k, self.k1, self.f = k, k1, torch.where(kk > 0, f, torch.zeros_like(f))
        self.pairs = []

        def keep(i, j, d, rr):
            t1, t2 = _rpy_real(a, rr, True)
            n = rr < 4.0
            ar = 4.0 / self.L
            o, g = _rpy_real(ar, rr, False), _rpy_real(ar, rr, True)
            t1, t2 = (torch.where(n, t + u - v, t) for t, u, v in zip((t1, t2), o, g))
            self.pairs.append((i, j, d, t1, t2 / rr))

        self.near(self.rc, keep)

    def apply(self, v):
        out = (1 - 6 / math.sqrt(math.pi) * self.a
               + 40 / (3 * math.sqrt(math.pi)) * self.a ** 3) * v
        F = torch.stack([torch.fft.rfftn(self.spread(v[:, d].contiguous())) for d in range(3)])
        kF = sum(self.k[..., d] * F[d] for d in range(3)) / self.k1
        for d in range(3):
            phi = torch.fft.irfftn(self.f * (F[d] - self.k[..., d] * kF), s=(self.K,) * 3)
            out[:, d] += self.gather(phi * self.K ** 3)
        for i, j, d, t1, t2 in self.pairs:
            q = t2 * (d * v[j]).sum(-1)
            out.index_add_(0, i, t1[:, None] * v[j] + q[:, None] * d)
        return out


def _exact_forces(c, x, y, z, q, qk):
    m = _Mesh(c, x, y, z)
    d = m.r.device
    f = torch.zeros_like(m.r)
    b = torch.arange(1, len(m.r), device=d)
    b = b[b % c["Nb"] != 0]
    v = m.r[b] - m.r[b - 1]
    s = v @ m.Hi.T
    v = (s - torch.round(s)) @ m.H.T
    t = (-30.0 / (1.0 - (v * v).sum(-1) / 9.0))[:, None] * v
    f.index_add_(0, b, t)
    f.index_add_(0, b - 1, -t)
    charge = torch.zeros(len(m.r), dtype=torch.float64, device=d)
    charge[torch.tensor(q, device=d).long()] = torch.tensor(qk, device=d)
    rc = min(10.0, 0.43 * m.L)
    beta, lb, energy = 3.5 / rc, 2.0, [0.0]

    def pair(i, j, dv, rr):
        r6 = (4.0 / rr) ** 3
        if c["flow"] == 0:
            co = torch.where(rr < 25.0, 12 / rr * (r6 * r6 - r6), 0 * rr)
        else:
            co = torch.where(rr < 5.03968, 48 / rr * (r6 * r6 - 0.5 * r6), 0 * rr)
        r = rr.sqrt()
        qq = lb * charge[i] * charge[j]
        ec = torch.erfc(beta * r) / r
        co = co + qq * (ec + 2 * beta / math.sqrt(math.pi) * torch.exp(-beta * beta * rr)) / rr
        energy[0] += float((0.5 * qq * ec).sum())
        f.index_add_(0, i, co[:, None] * dv)

    m.near(rc, pair)
    k, kk, bb = m.waves()
    G = 4 * math.pi * lb / (m.L ** 3 * kk) * torch.exp(-kk / (4 * beta * beta)) * bb
    G[0, 0, 0] = 0.0
    S = torch.fft.rfftn(m.spread(charge))
    twice = torch.full((m.K // 2 + 1,), 2.0, device=d, dtype=torch.float64)
    twice[0] = 1.0
    if m.K % 2 == 0:
        twice[-1] = 1.0
    energy[0] += float((0.5 * twice * G * S.abs().square()).sum())
    energy[0] -= lb * beta / math.sqrt(math.pi) * float((charge ** 2).sum())
    energy[0] -= math.pi * lb * float(charge.sum()) ** 2 / (2 * m.L ** 3 * beta * beta)
    phi = torch.fft.irfftn(G * S, s=(m.K,) * 3) * m.K ** 3
    du = torch.stack([m.gather(phi, a) for a in range(3)], 1)
    f -= charge[:, None] * m.K * (du @ m.Hi)
    return dict(forces=f.T.contiguous(), energy=energy[0])


def _exact_network(c, s, x, y, z):
    """Loss and gradient of the network (12 nearest beads within 6, 16 radial
    features, three layers of width 64), operands not rounded."""
    m = _Mesh(c, x, y, z)
    N, d = len(m.r), m.r.device
    near = [[], [], []]
    m.near(6.0, lambda i, j, dv, rr: [a.append(b) for a, b in zip(near, (i, dv, rr.sqrt()))])
    js = []
    m.near(6.0, lambda i, j, dv, rr: js.append(j))
    i, dv, r, j = torch.cat(near[0]), torch.cat(near[1]), torch.cat(near[2]), torch.cat(js)
    order = torch.argsort(r, stable=True)
    order = order[torch.argsort(i[order], stable=True)]
    i, dv, r, j = i[order], dv[order], r[order], j[order]
    n = torch.bincount(i, minlength=N)
    rank = torch.arange(len(i), device=d) - (torch.cumsum(n, 0) - n)[i]
    keep = rank < 12
    i, dv, r, j, rank = i[keep], dv[keep], r[keep], j[keep], rank[keep]
    at = i * 12 + rank
    nbr = torch.full((N * 12,), -1, device=d, dtype=torch.long).index_put_((at,), j).reshape(N, 12)
    n3 = torch.zeros(N * 12, 3, device=d, dtype=torch.float64).index_put_((at,), dv / r[:, None])
    n3 = n3.reshape(N, 12, 3)
    mu = 2.0 + 4.0 * torch.arange(16, device=d, dtype=torch.float64) / 15
    rb = torch.zeros(N * 12, 16, device=d, dtype=torch.float64)
    rb = rb.index_put_((at,), torch.exp(-0.5 * ((r[:, None] - mu) / 0.35) ** 2)).reshape(N, 12, 16)
    w = torch.tensor(np.asarray(s["w"], np.float64), device=d).requires_grad_()
    P, o = {}, 0
    for name, shape in B.MPNN_LAYOUT:
        size = int(np.prod(shape))
        P[name] = w[o:o + size].reshape(shape)
        o += size
    silu = torch.nn.functional.silu
    mask = (nbr >= 0).double()
    e = silu(rb @ P["W1"].T + P["b1"])
    h = silu((mask[..., None] * e).sum(1) / 12 @ P["W2"].T + P["b2"])
    hn = (h[nbr.clamp(min=0)] * mask[..., None]).sum(1) / 12
    u = silu(torch.cat([hn, h], 1) @ P["W34"].T + P["b3"])
    a = torch.exp((u @ P["wa"] + P["ca"][0]).clamp(-4, 4))
    t = ((u * P["wb"])[:, None, :] * e).sum(-1) + P["cb"][0]
    co = torch.tanh(t) * (0.5 / 12) * mask
    zz = torch.tensor(s["z"], device=d).reshape(N, 3)
    tt = torch.tensor(s["t"], device=d).reshape(N, 3)
    Gz = a[:, None] * (zz + (co[..., None] * n3 * (n3 * zz[:, None, :]).sum(-1, True)).sum(1))
    loss = ((Gz - tt) ** 2).sum() / N
    loss.backward()
    return dict(loss=float(loss), grad=w.grad)


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("steps", "reference", "hop"):
        return None
    x, y, z, q, qk, r = _system(c, seed)
    N = len(x)
    if kind == "forces":
        return _exact_forces(c, x, y, z, q, qk)
    if kind == "network":
        w = B.mpnn_init(seed) + r.normal(0, 0.05, B.mpnn_param_count()).astype(np.float32)
        zz = r.normal(size=3 * N)
        return _exact_network(c, dict(w=w, z=zz, t=zz + 0.3 * r.normal(size=3 * N)), x, y, z)
    M = _Mobility(c, x, y, z)
    if kind == "product":
        V = torch.tensor(r.normal(size=(c["k"], 3 * N)), device=M.r.device)
        return torch.stack([M.apply(v.reshape(N, 3)).reshape(-1) for v in V])
    v = torch.tensor(r.normal(size=3 * N), device=M.r.device)
    if kind == "rebuild":
        return M.apply(v.reshape(N, 3)).reshape(-1)
    cols = torch.eye(3 * N, device=M.r.device, dtype=torch.float64)
    A = torch.stack([M.apply(e.reshape(N, 3)).reshape(-1) for e in cols], 1)
    lam, U = torch.linalg.eigh(0.5 * (A + A.T))
    return U @ (lam.clamp(min=0).sqrt() * (U.T @ v))
