// Charge-hopping Monte Carlo with the reference's sequential sweep semantics.
//
// chargeHop (shear/src/main26.c:1926-2390) visits the charges in order; each
// trial draws one uniform, looks for the first bead (by index, excluding the
// charge's own bead and its index neighbours) within |NID|^2 < 4.41, proposes
// a move from the draw, and accepts with a Metropolis test on
// exp(-barrier - (E_final - E_initial)/2), where E_initial is the
// Debye-Hueckel energy at the start of the sweep (never refreshed) and
// E_final the energy with the trial move.  The reference recomputes E_final
// over all bead pairs for every trial (O(N^2) each); here E_final is carried
// incrementally, E_final = E_current + sum over the other charges of
// U(target, o) - U(source, o), which is the same quantity with a different
// summation order.
//
// Only the decisions are sequential.  A charge moves at most once in a sweep,
// at its own turn, so its source, the first bead near it and with them its
// three possible targets (c + 1, c - 1, that bead) are known beforehand.  The
// charges are taken 32 at a time: k_hop_window forms, with one CTA per charge,
// the energy change and the occupancy of each target for the sites at the
// window's start, and what each possible move of an earlier charge of the
// window adds to it; k_hop_decide then runs the window's trials in order with
// one warp, lane k holding charge k's three targets, so that a trial is its
// draws (the same, in the same order, as the reference), its Metropolis test
// and, when accepted, three table rows added to the later lanes.
#include <math.h>
#include <stddef.h>

#include "bd_ctx.cuh"
#include "bd_cell.cuh"

#define CU(call) BD_CU(call)

static const int kHopWin = 32;  // charges per window: one per lane of the deciding warp

__device__ __forceinline__ double dh_pair(const Lat& l, double xa, double ya, double za,
                                          double xb, double yb, double zb, double lambda_b,
                                          double kappa_d) {
  double vx, vy, vz;
  min_image(l, subx(xa, xb), subx(ya, yb), subx(za, zb), vx, vy, vz);
  double r = sqrt(rr3(vx, vy, vz));
  return (lambda_b / r) * exp(-kappa_d * r);
}

// Per-charge partial sums of the sweep's starting energy (pairs o > k).
__global__ void k_dh_energy_rows(Lat l, const double4* __restrict__ cq, int nch, double lambda_b,
                                 double kappa_d, double* rowsum) {
  int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (k >= nch) return;
  double4 a = cq[k];
  double s = 0;
  for (int o = k + 1 + lane; o < nch; o += 32) {
    double4 b = cq[o];
    s += a.w * b.w * dh_pair(l, a.x, a.y, a.z, b.x, b.y, b.z, lambda_b, kappa_d);
  }
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) rowsum[k] = s;
}

// Fixed-order block sum (every thread receives the total).
__device__ double block_sum(double v, double* sh) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    double x = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    if (lane == 0) sh[32] = x;
  }
  __syncthreads();
  return sh[32];
}

// First bead by index within |NID(c,j)|^2 < 4.41 of each charge, excluding
// c-1, c, c+1 (N: none); a warp per charge, 32 beads at a time.
__global__ void __launch_bounds__(256) k_hop_first(Lat l, const double* __restrict__ rx,
                                                   const double* __restrict__ ry,
                                                   const double* __restrict__ rz, int N, int nch,
                                                   const int* __restrict__ track,
                                                   int* __restrict__ first) {
  int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= nch) return;
  int c = track[k], found = N;
  double xc = rx[c], yc = ry[c], zc = rz[c];
  for (int base = 0; base < N; base += 32) {
    int j = base + lane;
    bool hit = false;
    if (j < N && j != c && j != c + 1 && j != c - 1) {
      double vx, vy, vz;
      min_image(l, subx(xc, rx[j]), subx(yc, ry[j]), subx(zc, rz[j]), vx, vy, vz);
      hit = rr3(vx, vy, vz) < 4.41;
    }
    unsigned m = __ballot_sync(0xffffffffu, hit);
    if (m) {
      found = base + __ffs(m) - 1;
      break;
    }
  }
  if (lane == 0) first[k] = found;
}

// A charge's source and its possible targets: the next and the previous bead
// of its chain and the first bead near it; -1 where there is none (chain ends,
// no bead near).
struct HopSites {
  int s[4];  // source, then the targets
};
__device__ __forceinline__ HopSites hop_sites(int c, int first, int N, int Nb) {
  HopSites h;
  h.s[0] = c;
  h.s[1] = (c == N - 1 || c % Nb == Nb - 1 || c == Nb - 1) ? -1 : c + 1;
  h.s[2] = (c - 1 < 0 || c == 0 || c % Nb == 0) ? -1 : c - 1;
  h.s[3] = first < N ? first : -1;
  return h;
}

// Scratch of a window: energy changes and occupancies of its charges' targets
// at the window's start, the table of what accepted moves add, the sweep's
// starting and current energy.
struct HopWin {
  double de[3 * kHopWin];                 // [target][charge]
  int occ[3 * kHopWin];
  double tab[kHopWin * 9 * kHopWin];      // [moved charge][its target][target][charge]
  double e_init, e_cur;
};
static_assert(offsetof(HopWin, tab) % 16 == 0, "the table is copied 16 bytes at a time");

struct HopArgs {
  Lat l;
  const double *rx, *ry, *rz;
  int N, Nb, nch;
  int* track;
  const int* first;
  const double* qk;
  double lambda_b, kappa_d;
  HopWin* win;
};

// One CTA per charge of the window.  The pair of a target with a charge that
// sits on it is left out everywhere: the trial is blocked while it sits there.
__global__ void __launch_bounds__(256) k_hop_window(HopArgs q, int k0) {
  __shared__ double red[8][3];
  __shared__ int redn[8][3];
  __shared__ double su[kHopWin][16];
  const int kk = blockIdx.x, k = k0 + kk, t = threadIdx.x;
  const HopSites h = hop_sites(q.track[k], q.first[k], q.N, q.Nb);
  double x[4], y[4], z[4];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    int b = max(h.s[a], 0);
    x[a] = q.rx[b];
    y[a] = q.ry[b];
    z[a] = q.rz[b];
  }
  const double qk = q.qk[k];
  double de[3] = {0, 0, 0};
  int occ[3] = {0, 0, 0};
  for (int o = t; o < q.nch; o += blockDim.x) {
    if (o == k) continue;
    int b = q.track[o];
    double xb = q.rx[b], yb = q.ry[b], zb = q.rz[b], qq = qk * q.qk[o];
    double uc = dh_pair(q.l, x[0], y[0], z[0], xb, yb, zb, q.lambda_b, q.kappa_d);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (h.s[a + 1] < 0) continue;
      double u = 0;
      if (b == h.s[a + 1])
        occ[a]++;
      else
        u = dh_pair(q.l, x[a + 1], y[a + 1], z[a + 1], xb, yb, zb, q.lambda_b, q.kappa_d);
      de[a] += qq * (u - uc);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++)
    for (int off = 16; off > 0; off >>= 1) {
      de[a] += __shfl_xor_sync(0xffffffffu, de[a], off);
      occ[a] += __shfl_xor_sync(0xffffffffu, occ[a], off);
    }
  if ((t & 31) == 0)
    for (int a = 0; a < 3; a++) {
      red[t >> 5][a] = de[a];
      redn[t >> 5][a] = occ[a];
    }
  // pairs with the sites of the window's earlier charges
  for (int e = t; e < 16 * kk; e += blockDim.x) {
    int m = e >> 4, a = (e >> 2) & 3, bb = e & 3;
    HopSites g = hop_sites(q.track[k0 + m], q.first[k0 + m], q.N, q.Nb);
    int sa = a == 0 ? h.s[0] : a == 1 ? h.s[1] : a == 2 ? h.s[2] : h.s[3];
    int sb = bb == 0 ? g.s[0] : bb == 1 ? g.s[1] : bb == 2 ? g.s[2] : g.s[3];
    double u = 0;
    if (sa >= 0 && sb >= 0 && sa != sb)
      u = dh_pair(q.l, q.rx[sa], q.ry[sa], q.rz[sa], q.rx[sb], q.ry[sb], q.rz[sb], q.lambda_b,
                  q.kappa_d);
    su[m][4 * a + bb] = u;
  }
  __syncthreads();
  if (t < 3) {
    double s = 0;
    int n = 0;
    for (int w = 0; w < 8; w++) {
      s += red[w][t];
      n += redn[w][t];
    }
    q.win->de[t * kHopWin + kk] = s;
    q.win->occ[t * kHopWin + kk] = n;
  }
  for (int e = t; e < 9 * kHopWin; e += blockDim.x) {
    int m = e / 9, om = (e % 9) / 3, ok = e % 3;
    double d = 0;
    if (m < kk)
      d = qk * q.qk[k0 + m] *
          (su[m][4 * (ok + 1) + om + 1] - su[m][4 * (ok + 1)] - su[m][om + 1] + su[m][0]);
    q.win->tab[e * kHopWin + kk] = d;
  }
}

// Energy change of moving charge k from c to c2 for the sites as they are, by
// one warp: for trials that the window's sums cannot give, a pair at distance
// zero among them (infinite terms that would cancel).
__device__ double hop_energy(const HopArgs& q, int k, int c, int c2) {
  double de = 0, qk = q.qk[k];
  for (int o = threadIdx.x & 31; o < q.nch; o += 32) {
    if (o == k) continue;
    int b = __ldcv(q.track + o);
    de += qk * q.qk[o] *
          (dh_pair(q.l, q.rx[c2], q.ry[c2], q.rz[c2], q.rx[b], q.ry[b], q.rz[b], q.lambda_b,
                   q.kappa_d) -
           dh_pair(q.l, q.rx[c], q.ry[c], q.rz[c], q.rx[b], q.ry[b], q.rz[b], q.lambda_b,
                   q.kappa_d));
  }
  for (int off = 16; off > 0; off >>= 1) de += __shfl_xor_sync(0xffffffffu, de, off);
  return de;
}

// The generator's next m <= 64 uniforms into u (unless null), by one warp; with
// keep its state is left as it was, else advanced by m.
__device__ void ran1_draws(Ran1* gs, uint4* next, int m, float* u, bool keep) {
  const int lane = threadIdx.x & 31;
  Ran1Warp r;
  if (r.load(gs)) {
    unsigned y0 = 0, y1 = 0;
    r.ahead(next);
    r.walk(next, m, y0, y1);
    if (u) {
      u[lane] = Ran1Warp::uniform(y0);
      u[32 + lane] = Ran1Warp::uniform(y1);
    }
    if (!keep) r.store(gs);
  } else if (lane == 0) {
    Ran1 g = *gs;
    for (int t = 0; t < m; t++) {
      float x = ran1_dev(g);
      if (u) u[t] = x;
    }
    if (!keep) *gs = g;
  }
  __syncwarp();
}

// The window's trials in order.  They use at most two uniforms each: 64 are
// drawn before the trials, and the generator is advanced by those used after
// them.  Bound by the trials' serial chain (test, exponential, table row):
// 15.5 us a window, k_hop_window 8; a sweep over 250 charges among 500 beads
// 0.2 ms, 0.73 ms with one block searching, testing and summing charge by
// charge.
__global__ void __launch_bounds__(256) k_hop_decide(HopArgs q, int k0,
                                                    const double* __restrict__ rowsum,
                                                    int* __restrict__ old, Ran1* rng,
                                                    double barrier, double barrier2, int* log) {
  extern __shared__ __align__(16) double tab[];  // filled 16 bytes at a time
  __shared__ double red[33];
  __shared__ uint4 next[64];
  __shared__ float u[64];
  __shared__ double ud[65];  // one past the last: read, not used, when x >= 1
  __shared__ int pick[64];   // target drawn with a bead near | without, 4 times
  const int t = threadIdx.x, w = min(kHopWin, q.nch - k0);
  double E_init, E_cur;
  if (k0 == 0) {
    double e0 = 0;
    for (int k = t; k < q.nch; k += blockDim.x) e0 += rowsum[k];
    E_init = q.nch > 1 ? block_sum(e0, red) : 0.0;
    E_cur = E_init;
  } else {
    E_init = q.win->e_init;
    E_cur = q.win->e_cur;
  }
  if (t < 32) {
    ran1_draws(rng, next, 2 * kHopWin, u, true);
    for (int e = t; e < 2 * kHopWin; e += 32) {
      double mm = (double)u[e];
      pick[e] = (mm < .33 ? 0 : mm > 0.66 ? 1 : 2) | (mm > .5 ? 0 : 4);
      ud[e] = mm;
    }
  } else {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(tab);
    for (int e = t - 32; e < w * 9 * kHopWin / 2; e += blockDim.x - 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e),
                   "l"(q.win->tab + 2 * e));
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  if (t >= 32) return;
  const int k = k0 + min(t, w - 1);
  const int c = q.track[k];
  const HopSites h = hop_sites(c, q.first[k], q.N, q.Nb);
  const bool near = h.s[3] >= 0;
  double de0 = q.win->de[t], de1 = q.win->de[kHopWin + t], de2 = q.win->de[2 * kHopWin + t];
  int oc0 = h.s[1] < 0 ? 1 : q.win->occ[t], oc1 = h.s[2] < 0 ? 1 : q.win->occ[kHopWin + t];
  int oc2 = q.win->occ[2 * kHopWin + t];
  int used = 0, did = 0, to = c, kind = 0;  // this lane's trial: log, target, move kind
  for (int kk = 0; kk < w; kk++) {
    const int pk = pick[used], opt_l = near ? pk & 3 : pk >> 2;
    const int tgt = opt_l == 0 ? c + 1 : opt_l == 1 ? c - 1 : h.s[3];
    const int occ = opt_l == 0 ? oc0 : opt_l == 1 ? oc1 : oc2;
    const double de_l = opt_l == 0 ? de0 : opt_l == 1 ? de1 : de2;
    const int test_l = near ? (opt_l == 2 ? 2 : 1) : 0;
    used++;
    const int info = __shfl_sync(0xffffffffu, opt_l | (test_l << 2) | ((occ > 0) << 4), kk);
    const int c2 = __shfl_sync(0xffffffffu, tgt, kk), c1 = __shfl_sync(0xffffffffu, c, kk);
    double de = __shfl_sync(0xffffffffu, de_l, kk);
    const int opt = info & 3, test = (info >> 2) & 3;
    if (t == kk) to = c2;
    if (info >> 4) continue;  // blocked: the log keeps no move kind
    double E_fin = 0.0;
    if (q.nch > 1) {
      if (!isfinite(de)) {
        if (t < kk && did == 1) q.track[k] = to;
        __syncwarp();
        de = hop_energy(q, k0 + kk, c1, c2);
      }
      E_fin = E_cur + de;
    }
    const double x = exp(-(test == 2 ? barrier2 : barrier) - 0.5 * (E_fin - E_init));
    const bool sure = 1 <= x, acc = sure || ud[used] <= x;
    used += !sure;
    if (t == kk) {
      did = acc ? 1 : 2;
      kind = test;
    }
    if (!acc) continue;
    E_cur = E_fin;
    const double* row = tab + (size_t)(3 * kk + opt) * 3 * kHopWin + t;
    de0 += row[0];
    de1 += row[kHopWin];
    de2 += row[2 * kHopWin];
    oc0 += (h.s[1] == c2) - (h.s[1] == c1);
    oc1 += (h.s[2] == c2) - (h.s[2] == c1);
    oc2 += (h.s[3] == c2) - (h.s[3] == c1);
  }
  if (t < w) {
    if (did) old[k] = c;
    if (did == 1) q.track[k] = to;
    log[3 * k] = did;
    log[3 * k + 1] = to;
    log[3 * k + 2] = kind;
  }
  ran1_draws(rng, next, used, nullptr, false);
  if (t == 0) {
    q.win->e_init = E_init;
    q.win->e_cur = E_cur;
  }
}

__global__ void k_charge_values(const double* __restrict__ q, const int* __restrict__ track,
                                int nch, double* qk) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nch) qk[k] = q[track[k]];
}

__global__ void k_clear_charges(int* flags, double* q, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) {
    flags[i] = 0;
    q[i] = 0.0;
  }
}

__global__ void k_scatter_charges(const int* __restrict__ track, const double* __restrict__ qk,
                                  int nch, int* flags, double* q) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nch) {
    flags[track[k]] = 1;
    q[track[k]] = qk[k];
  }
}

__global__ void k_gather_charges_mc(const double* __restrict__ rx, const double* __restrict__ ry,
                                    const double* __restrict__ rz, const double* __restrict__ q,
                                    const int* __restrict__ track, int nch, double4* out) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nch) {
    int i = track[k];
    out[k] = make_double4(rx[i], ry[i], rz[i], q[i]);
  }
}

namespace bd {

size_t hop_win_bytes() { return sizeof(HopWin); }

int charge_hop_parallel(bd_ctx* c);

int charge_hop(bd_ctx* c) {
  if (c->nch == 0) return BD_OK;
  if (c->t % (unsigned long)c->p.MStep != 0) return BD_OK;
  if (c->p.hop == BD_HOP_PARALLEL) return charge_hop_parallel(c);
  int nch = c->nch, N = c->N;
  // scratch in dE (8 N doubles): [0, 4 nch) gathered (x,y,z,q); then row
  // sums; then qk; then the first bead near each charge
  double4* cq = (double4*)c->dE;
  double* rowsum = c->dE + 4 * (size_t)nch;
  double* qk = rowsum + nch;
  int* first = (int*)(qk + nch);
  Lat l = c->lat;
  int treal = (int)(c->t % (unsigned long)c->tp);
  l.treal = treal;
  l.delx = c->p.edot * treal * c->p.dt;
  c->launches++;
  k_charge_values<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->q, c->track, nch, qk);
  c->launches++;
  k_gather_charges_mc<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->rx, c->ry, c->rz, c->q, c->track,
                                                             nch, cq);
  c->launches++;
  k_dh_energy_rows<<<(nch * 32 + 255) / 256, 256, 0, c->stream>>>(l, cq, nch, c->p.lambda_b,
                                                                   c->kappa_d, rowsum);
  HopArgs q;
  q.l = l;
  q.rx = c->rx;
  q.ry = c->ry;
  q.rz = c->rz;
  q.N = N;
  q.Nb = c->Nb;
  q.nch = nch;
  q.track = c->track;
  q.first = first;
  q.qk = qk;
  q.lambda_b = c->p.lambda_b;
  q.kappa_d = c->kappa_d;
  q.win = (HopWin*)c->hop_win;
  const int smem = 8 * 9 * kHopWin * kHopWin;
  CU(cudaFuncSetAttribute(k_hop_decide, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  prof_begin(c, BD_PROF_HOP);
  c->launches++;
  k_hop_first<<<(nch * 32 + 255) / 256, 256, 0, c->stream>>>(l, c->rx, c->ry, c->rz, N, nch,
                                                             c->track, first);
  for (int k0 = 0; k0 < nch; k0 += kHopWin) {
    c->launches += 2;
    k_hop_window<<<std::min(kHopWin, nch - k0), 256, 0, c->stream>>>(q, k0);
    k_hop_decide<<<1, 256, smem, c->stream>>>(q, k0, rowsum, c->old, c->rng, c->p.barrier,
                                              c->p.barrier2, c->hoplog);
  }
  prof_end(c, BD_PROF_HOP);
  c->launches++;
  k_clear_charges<<<(N + 255) / 256, 256, 0, c->stream>>>(c->cflags, c->q, N);
  c->launches++;
  k_scatter_charges<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->track, qk, nch, c->cflags, c->q);
  return launch_ok(c);
}

}  // namespace bd

// ---------------------------------------------------------------------------
// Parallel sweep on independent sets (no reference counterpart).
//
// The charges are binned into cells of the Gauss-reduced cell at least R
// wide (R = hop_radius, default 3 Debye lengths), with an even number of
// cells per direction; the parity of the three cell indices gives eight
// colours, and cells of one colour are at least R apart.  A sweep runs the
// eight colours in turn; within a colour the trials' energies against the charges at
// the colour's start are formed at once, and a warp per cell then visits its charges
// in index order, each exactly once.  A trial follows the reference's
// proposal rules (partner search, chain ends, occupancy, the two barriers) and
// accepts with min(1, exp(-barrier - dE/2)) (the reference's factor, without
// its stale starting energy), dE the energy change of the move against every
// other charge: with Debye-Hueckel electrostatics the reference's screened
// pair energy; with Ewald electrostatics the unscreened energy the forces
// use, in FP64:
//   dE = q sum_o q_o [erfc(beta r)/r]_a^b   (real space, within the cutoff)
//      + q [Phi0(b) - Phi0(a)]               (mesh reciprocal potential of all
//                                              charges at the colour's start)
//      - q^2 [G(b - a) - G(0)]               (the moved charge's own term)
//      + q sum_j q_j [G(b-b_j) - G(b-a_j) - G(a-b_j) + G(a-a_j)]
//                                            (charges of the own cell moved
//                                              earlier in the colour, a_j -> b_j)
// with G(r) = lambda_B erf(beta r)/r + r^T Q r the reciprocal pair term near
// the origin (Q the quadratic form of its periodic remainder, from the
// lattice's k-space sum, (2 pi lambda_B / 3 V) I for a cubic cell; the rest is
// O(r^4 / L^5); G(0) = 2 beta lambda_B/sqrt(pi)).  The other
// charges are taken at their sites at the start of the colour, those of the
// own cell at their current sites; a move therefore ignores only the change
// of its interaction with charges moved in the same colour in other cells,
// which are at least R away: the second difference of the pair energy over
// both hops, |dU| <= 2 lambda_B d^2 / R^3 per pair (hop distance d <= 2.1),
// 0.005 kT at R = 15 for the bare Coulomb energy, less when screened.  The
// draws are Philox4x32-10
// counters (charge, sweep, purpose) under philox_seed, so a sweep does not
// depend on the launch order.  The partner is the first bead of the charge's
// Verlet row (sorted ascending, radius 6 > 2.1 plus twice the skin) within
// |NID|^2 < 4.41, as the reference's scan over all beads finds it.

namespace {

constexpr int kHopCellCap = 8192;

struct HGeom {
  int n[3];
};

__device__ __forceinline__ double philox_u01(int k, unsigned long long sweep, int tag,
                                             unsigned long long seed) {
  uint4 c = make_uint4((uint32_t)k, (uint32_t)sweep, (uint32_t)(sweep >> 32),
                       0x4d430000u | (uint32_t)tag);
  uint4 x = philox4x32_10(c, make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  return (double)(((unsigned long long)(x.x >> 5) << 26) | (x.y >> 6)) *
         (1.0 / 9007199254740992.0);
}

__global__ void k_hop_cells(Cell cell, HGeom g, const double* __restrict__ rx,
                            const double* __restrict__ ry, const double* __restrict__ rz,
                            const int* __restrict__ track, int nch, double cr, double sr,
                            int* cell_of, int* count) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nch) return;
  int b = track[k];
  double x = rx[b] * cr - ry[b] * sr, y = rx[b] * sr + ry[b] * cr, s[3];
  frac_of(cell, x, y, rz[b], s);
  int cd[3];
  for (int d = 0; d < 3; d++) {
    double sd = s[d] - floor(s[d]);
    int c = (sd >= 0.0 && sd <= 1.0) ? (int)(sd * g.n[d]) : 0;
    cd[d] = c >= g.n[d] ? g.n[d] - 1 : c;
  }
  int c = (cd[0] * g.n[1] + cd[1]) * g.n[2] + cd[2];
  cell_of[k] = c;
  atomicAdd(&count[c], 1);
}

__global__ void k_hop_scan(int ncell, int* count, int* start) {
  __shared__ int part[1024];
  int t = threadIdx.x, nt = blockDim.x;
  int per = (ncell + nt - 1) / nt, lo = t * per, hi = min(ncell, lo + per), s = 0;
  for (int c = lo; c < hi; c++) s += count[c];
  part[t] = s;
  __syncthreads();
  for (int o = 1; o < nt; o <<= 1) {
    int v = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int b = part[t] - s;
  for (int c = lo; c < hi; c++) {
    start[c] = b;
    b += count[c];
    count[c] = 0;
  }
  if (t == nt - 1) start[ncell] = part[t];
}

// One warp per cell lists its charges in increasing index (a fixed order):
// 256 cell numbers are read at a time and the matches placed by ballot.
// Latency-bound; with one thread per cell it took 682 us for 25 000 charges.
__global__ void __launch_bounds__(128) k_hop_fill(const int* __restrict__ cell_of,
                                                  const int* __restrict__ start, int ncell,
                                                  int nch, int* __restrict__ idx) {
  int c = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= ncell) return;
  int p = start[c];
  const int end = start[c + 1];
  for (int k0 = 0; k0 < nch && p < end; k0 += 256) {
    int v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      int k = k0 + 32 * u + lane;
      v[u] = k < nch ? cell_of[k] : -1;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      unsigned hit = __ballot_sync(0xffffffffu, v[u] == c);
      if (v[u] == c) idx[p + __popc(hit & ((1u << lane) - 1u))] = k0 + 32 * u + lane;
      p += __popc(hit);
    }
  }
}

// The Ewald energy terms of a trial (P > 0): the lab-frame reduced cell, the
// stored-frame rotation, the reciprocal potential on the mesh, the split.
struct HopEwald {
  Cell cell;
  double cr, sr;
  const double* phi;
  const double* Q;  // quadratic form of the reciprocal pair term's periodic remainder
  int K;
  double beta, rc2, lambda_b;
};

__device__ __forceinline__ void hop_lab(const HopEwald& ew, double x, double y, double& lx,
                                        double& ly) {
  lx = x * ew.cr - y * ew.sr;
  ly = x * ew.sr + y * ew.cr;
}

// Minimum image of d in the reduced cell.
__device__ __forceinline__ void hop_minimg(const HopEwald& ew, double& dx, double& dy,
                                           double& dz) {
  double s[3];
  frac_of(ew.cell, dx, dy, dz, s);
  for (int d = 0; d < 3; d++) s[d] -= rint(s[d]);
  const double* H = ew.cell.H;
  dx = H[0] * s[0] + H[1] * s[1] + H[2] * s[2];
  dy = H[3] * s[0] + H[4] * s[1] + H[5] * s[2];
  dz = H[6] * s[0] + H[7] * s[1] + H[8] * s[2];
}

__device__ __forceinline__ double hop_rr(const HopEwald& ew, double dx, double dy, double dz) {
  hop_minimg(ew, dx, dy, dz);
  return dx * dx + dy * dy + dz * dz;
}

// Two charges' sites below this squared distance are one site: the trial's
// target, occupied at the colour's start by a charge that has moved away since.
// The pair term of that site is left out of both the sum at the colour's start
// and the correction for the move, whose difference it would cancel from.
constexpr double kSameSite = 1e-16;

__device__ __forceinline__ double hop_dh(const Lat& l, const double4& a, const double4& b,
                                         double lambda_b, double kappa_d) {
  double vx, vy, vz;
  min_image(l, subx(a.x, b.x), subx(a.y, b.y), subx(a.z, b.z), vx, vy, vz);
  double rr = rr3(vx, vy, vz);
  if (rr < kSameSite) return 0.0;
  double r = sqrt(rr);
  return (lambda_b / r) * exp(-kappa_d * r);
}

// Real-space pair term lambda_B erfc(beta r)/r within the cutoff.
__device__ __forceinline__ double hop_real(const HopEwald& ew, double dx, double dy, double dz) {
  double rr = hop_rr(ew, dx, dy, dz);
  if (rr >= ew.rc2 || rr < kSameSite) return 0.0;
  double r = sqrt(rr);
  return ew.lambda_b * erfc(ew.beta * r) / r;
}

// Reciprocal pair term near the origin, G(r) = lambda_B erf(beta r)/r + r^T Q r
// (the Gaussian-screened part and the quadratic term of the periodic remainder;
// its constant cancels in every difference, its O(r^4 / L^5) rest is left
// out); G(0) = 2 beta lambda_B / sqrt(pi).
__device__ __forceinline__ double hop_recip(const HopEwald& ew, double dx, double dy, double dz) {
  hop_minimg(ew, dx, dy, dz);
  double rr = dx * dx + dy * dy + dz * dz, r = sqrt(rr);
  if (r <= 1e-12) return ew.lambda_b * 2.0 * ew.beta / sqrt(M_PI);
  const double* Q = ew.Q;
  double quad = Q[0] * dx * dx + Q[3] * dy * dy + Q[5] * dz * dz +
                2.0 * (Q[1] * dx * dy + Q[2] * dx * dz + Q[4] * dy * dz);
  return ew.lambda_b * erf(ew.beta * r) / r + quad;
}

// hop_real + hop_recip: within the cutoff the split's two halves add up to
// lambda_B / r, so only pairs beyond it need an error function.
__device__ __forceinline__ double hop_full(const HopEwald& ew, double dx, double dy, double dz) {
  hop_minimg(ew, dx, dy, dz);
  double rr = dx * dx + dy * dy + dz * dz;
  if (rr < kSameSite) return ew.lambda_b * 2.0 * ew.beta / sqrt(M_PI);
  const double* Q = ew.Q;
  double quad = Q[0] * dx * dx + Q[3] * dy * dy + Q[5] * dz * dz +
                2.0 * (Q[1] * dx * dy + Q[2] * dx * dz + Q[4] * dy * dz);
  double r = sqrt(rr), f = ew.lambda_b / r;
  return (rr >= ew.rc2 ? f * erf(ew.beta * r) : f) + quad;
}

// A colour's sweep in two parts.  Positions are fixed during a sweep and each
// charge is tried once, so its proposal is known before the sweep starts
// (k_hop_propose), and the part of its energy change that refers to the
// charges at their sites at the colour's start needs no other trial's outcome
// (k_hop_base: every trial of the colour at once, a warp each, the real-space
// sum over the charges of the neighbouring coulomb cells only).  What is left
// in order (k_hop_accept, a warp per cell) is the occupancy test, the
// correction for the cell's own charges that moved earlier in the colour, and
// the acceptance.  Latency-bound in the ordered part.  With one CTA doing a
// whole trial at a time over all the charges a colour took 3.30 ms at 25 000
// charges; now 0.07 ms and 0.11 ms, and 0.13 ms for the mesh and the cells.

// Target bead of each charge's trial and its kind: bits 0-1 the reference's
// test index, bit 2 set for a blocked move.  One warp per charge.
__global__ void __launch_bounds__(256)
    k_hop_propose(Lat l, const double* __restrict__ rx, const double* __restrict__ ry,
                  const double* __restrict__ rz, int N, int Nb, int nch,
                  const int* __restrict__ track, const int* __restrict__ nb_count,
                  const int* __restrict__ nb_rows, int maxnb, unsigned long long seed,
                  unsigned long long sweep, int* target, int* kind) {
  int k = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= nch) return;
  int c = track[k], nr = min(nb_count[c], maxnb), first = -1;
  double xc = rx[c], yc = ry[c], zc = rz[c];
  // the rows are sorted: the first hit is the lowest bead index
  for (int e0 = 0; e0 < nr && first < 0; e0 += 32) {
    int j = e0 + lane < nr ? nb_rows[(size_t)c * maxnb + e0 + lane] : c;
    bool in = false;
    if (j != c && j != c + 1 && j != c - 1) {
      double vx, vy, vz;
      min_image(l, subx(xc, rx[j]), subx(yc, ry[j]), subx(zc, rz[j]), vx, vy, vz);
      in = rr3(vx, vy, vz) < 4.41;
    }
    unsigned hit = __ballot_sync(0xffffffffu, in);
    if (hit) first = __shfl_sync(0xffffffffu, j, __ffs(hit) - 1);
  }
  if (lane) return;
  double mm = philox_u01(k, sweep, 0, seed);
  int c2, test = 0;
  if (first >= 0) {
    test = mm < .33 || mm > 0.66 ? 1 : 2;
    c2 = mm < .33 ? c + 1 : mm > 0.66 ? c - 1 : first;
  } else {
    c2 = mm > .5 ? c + 1 : c - 1;
  }
  bool block = test == 2 ? false
               : c2 > c  ? (c == N - 1 || c % Nb == Nb - 1 || c == Nb - 1)
                         : (c2 < 0 || c == 0 || c % Nb == 0);
  target[k] = c2;
  kind[k] = test | (block ? 4 : 0);
}

__device__ __forceinline__ bool hop_in_colour(const HGeom& g, int cell, int colour) {
  int cz = cell % g.n[2], cy = (cell / g.n[2]) % g.n[1], cx = cell / (g.n[1] * g.n[2]);
  return (((g.n[0] > 1 ? cx & 1 : 0) << 2) | ((g.n[1] > 1 ? cy & 1 : 0) << 1) |
          (g.n[2] > 1 ? cz & 1 : 0)) == colour;
}

// The colour's trials (entry q of the cells' lists): energy change against the
// other charges at their sites at the colour's start (cq; cells ccn, ranges
// ccs, charges in cell order cci and ccp), with Ewald electrostatics the mesh
// and own terms too.  P = 0: Debye-Hueckel; P = 4, 6, 8: Ewald, B-spline order.
template <int P>
__global__ void __launch_bounds__(256)
    k_hop_base(Lat l, HGeom g, int colour, const double* __restrict__ rx,
               const double* __restrict__ ry, const double* __restrict__ rz, int nch,
               const int* __restrict__ idx, const int* __restrict__ cell_of,
               const int* __restrict__ track, const double* __restrict__ qk,
               const int* __restrict__ target, const int* __restrict__ kind,
               const double4* __restrict__ cq, HGeom ccg, const int* __restrict__ ccs,
               const int* __restrict__ cci, const double4* __restrict__ ccp, double lambda_b,
               double kappa_d, HopEwald ew, double* de0) {
  __shared__ CandList s_list[8];
  __shared__ double s_w[8][2][3][P > 0 ? P : 1];  // spline weights of both sites
  __shared__ int s_base[8][2][3];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * 8 + wl;
  if (q >= nch) return;
  const int k = idx[q];
  if (!hop_in_colour(g, cell_of[k], colour) || (kind[k] & 4)) return;
  const int c = track[k], c2 = target[k];
  const double xc = rx[c], yc = ry[c], zc = rz[c], x2 = rx[c2], y2 = ry[c2], z2 = rz[c2];
  const double qme = qk[k];
  double de = 0;
  if constexpr (P == 0) {
    for (int o = lane; o < nch; o += 32) {
      if (o == k) continue;
      double4 b = cq[o];
      de += qme * b.w *
            (hop_dh(l, make_double4(x2, y2, z2, 0.0), b, lambda_b, kappa_d) -
             hop_dh(l, make_double4(xc, yc, zc, 0.0), b, lambda_b, kappa_d));
    }
  } else {
    double sx[2], sy[2], sz[2] = {zc, z2};
    hop_lab(ew, xc, yc, sx[0], sy[0]);
    hop_lab(ew, x2, y2, sx[1], sy[1]);
#pragma unroll
    for (int pt = 0; pt < 2; pt++) {
      int cd[3];
      cell_of_pos(ew.cell, ccg.n, sx[pt], sy[pt], sz[pt], cd);
      int total = s_list[wl].open(ccg.n, cd, ccs), cl = 0;
      double sum = 0;
      for (int m = lane; m < total; m += 32) {
        int at = s_list[wl].at(m, cl);
        double4 o = ccp[at];
        double t = hop_real(ew, sx[pt] - o.x, sy[pt] - o.y, sz[pt] - o.z);
        if (cci[at] != k) sum += o.w * t;
      }
      de += pt ? qme * sum : -qme * sum;
    }
    // spline weights of the two sites (lane 3 pt + d: site pt, direction d)
    if (lane < 6) {
      int pt = lane / 3, d = lane % 3;
      double sv[3];
      frac_of(ew.cell, pt ? sx[1] : sx[0], pt ? sy[1] : sy[0], pt ? sz[1] : sz[0], sv);
      double sd = d == 0 ? sv[0] : d == 1 ? sv[1] : sv[2];
      double u = (sd - floor(sd)) * ew.K;
      if (!(u >= 0.0 && u <= (double)ew.K)) u = 0.0;
      int fl = (int)floor(u);
      double f = u - fl;
      if (fl >= ew.K) fl -= ew.K;
      s_base[wl][pt][d] = fl;
      double wv[P];
      bspline_t<P>(f, wv);
#pragma unroll
      for (int a = 0; a < P; a++) s_w[wl][pt][d][a] = wv[a];
    }
    __syncwarp();
    // q [Phi0(b) - Phi0(a)] from the mesh
    constexpr int P3 = P * P * P;
    const int K = ew.K;
#pragma unroll 4
    for (int e = lane; e < 2 * P3; e += 32) {
      int pt = e / P3, m = e - pt * P3;
      int cc = m % P, bb = (m / P) % P, aa = m / (P * P);
      int g0 = s_base[wl][pt][0] - aa, g1 = s_base[wl][pt][1] - bb, g2 = s_base[wl][pt][2] - cc;
      g0 += g0 < 0 ? K : 0;
      g1 += g1 < 0 ? K : 0;
      g2 += g2 < 0 ? K : 0;
      double v = s_w[wl][pt][0][aa] * s_w[wl][pt][1][bb] * s_w[wl][pt][2][cc] *
                 ew.phi[((size_t)g0 * K + g1) * K + g2];
      de += pt ? qme * v : -qme * v;
    }
    // the moved charge's own reciprocal term
    if (lane == 0)
      de -= qme * qme * (hop_recip(ew, sx[1] - sx[0], sy[1] - sy[0], z2 - zc) -
                         hop_recip(ew, 0, 0, 0));
  }
  for (int o = 16; o > 0; o >>= 1) de += __shfl_xor_sync(0xffffffffu, de, o);
  if (lane == 0) de0[q] = de;
}

// A cell's trials in index order, one warp: 32 trials' data at a time in
// shared memory; moved holds the cell's accepted moves of this colour, two
// double4 each ((a, q), (b, -)), from entry start[cell] on.
template <int P>
__global__ void __launch_bounds__(32)
    k_hop_accept(Lat l, HGeom g, int colour, const double* __restrict__ rx,
                 const double* __restrict__ ry, const double* __restrict__ rz,
                 const int* __restrict__ start, const int* __restrict__ idx,
                 const double* __restrict__ qk, const int* __restrict__ target,
                 const int* __restrict__ kind_of, const double* __restrict__ de0, int* track,
                 int* old, int* flags, double4* moved, double lambda_b, double kappa_d,
                 double barrier, double barrier2, unsigned long long seed,
                 unsigned long long sweep, int* log, double* hop_de, HopEwald ew) {
  const int cell = blockIdx.x, lane = threadIdx.x;
  if (!hop_in_colour(g, cell, colour)) return;
  __shared__ double4 s_a[32], s_b[32];
  const int q0 = start[cell], q1 = start[cell + 1];
  moved += 2 * (size_t)q0;
  int nm = 0;
  for (int qb = q0; qb < q1; qb += 32) {
    const int nq = min(32, q1 - qb);
    int k = 0, c = 0, c2 = 0, kind = 4, taken = 1;
    double d0 = 0, u2 = 0, bar = 0;
    if (lane < nq) {
      k = idx[qb + lane];
      c = track[k];
      c2 = target[k];
      kind = kind_of[k];
      if (!(kind & 4)) {
        taken = flags[c2];  // occupied target
        d0 = de0[qb + lane];
        u2 = philox_u01(k, sweep, 1, seed);
        bar = (kind & 3) == 2 ? barrier2 : barrier;
        double ax = rx[c], ay = ry[c], bx = rx[c2], by = ry[c2];
        if constexpr (P > 0) {
          hop_lab(ew, rx[c], ry[c], ax, ay);
          hop_lab(ew, rx[c2], ry[c2], bx, by);
        }
        s_a[lane] = make_double4(ax, ay, rz[c], qk[k]);
        s_b[lane] = make_double4(bx, by, rz[c2], 0.0);
      }
    }
    __syncwarp();
    for (int u = 0; u < nq; u++) {
      if (__shfl_sync(0xffffffffu, taken, u)) {
        if (lane == u) {
          log[3 * k] = 0;
          log[3 * k + 1] = c2;
          log[3 * k + 2] = 0;
          hop_de[k] = __longlong_as_double(0x7ff8000000000000LL);  // no trial energy
        }
        continue;
      }
      const double4 a = s_a[u], b = s_b[u];
      // four pair terms per moved charge, a lane each: + (b, b_j) - (b, a_j)
      // - (a, b_j) + (a, a_j)
      double corr = 0;
      for (int e = lane; e < 4 * nm; e += 32) {
        const int m = e >> 2;
        const double4 aj = moved[2 * m], o = e & 1 ? aj : moved[2 * m + 1], p = e & 2 ? a : b;
        double t;
        if constexpr (P == 0)
          t = hop_dh(l, p, o, lambda_b, kappa_d);
        else
          t = hop_full(ew, p.x - o.x, p.y - o.y, p.z - o.z);
        corr += (e & 3) == 0 || (e & 3) == 3 ? aj.w * t : -aj.w * t;
      }
      if (nm > 0)
        for (int o = 16; o > 0; o >>= 1) corr += __shfl_xor_sync(0xffffffffu, corr, o);
      int acc = 0;
      if (lane == u) {
        double de = d0 + a.w * corr;
        hop_de[k] = de;
        double x = exp(-bar - 0.5 * de);
        acc = (1 <= x) ? 1 : (u2 <= x);
        old[k] = c;
        if (acc) {
          flags[c] = 0;
          flags[c2] = 1;
          track[k] = c2;
        }
        log[3 * k] = acc ? 1 : 2;
        log[3 * k + 1] = c2;
        log[3 * k + 2] = kind & 3;
      }
      if (__shfl_sync(0xffffffffu, acc, u)) {
        int was = __shfl_sync(0xffffffffu, c, u), now = __shfl_sync(0xffffffffu, c2, u);
        if (!(kind & 4)) taken = c2 == now ? 1 : c2 == was ? 0 : taken;
        if (lane == 0) {
          moved[2 * nm] = a;
          moved[2 * nm + 1] = b;
        }
        nm++;
        __syncwarp();
      }
    }
    __syncwarp();
  }
}

// (x, y, z, q) of each charge at its current site, in track order.
__global__ void k_gather_sites(const double* __restrict__ rx, const double* __restrict__ ry,
                               const double* __restrict__ rz, const int* __restrict__ track,
                               const double* __restrict__ qk, int nch, double4* cq) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nch) return;
  int b = track[k];
  cq[k] = make_double4(rx[b], ry[b], rz[b], qk[k]);
}

}  // namespace

namespace bd {

int charge_hop_parallel(bd_ctx* c) {
  int nch = c->nch, N = c->N;
  if (!c->hop_cells) {
    CU(cudaMalloc(&c->hop_cells, 4 * ((size_t)3 * N + 2 * (kHopCellCap + 1))));
    c->bytes += 4 * ((size_t)3 * N + 2 * (kHopCellCap + 1));
    CU(cudaMemsetAsync(c->hop_cells, 0, 4 * ((size_t)3 * N + 2 * (kHopCellCap + 1)), c->stream));
  }
  if (!c->hop_work) {
    CU(cudaMalloc(&c->hop_work, 8 * (16 * (size_t)N + 8)));
    c->bytes += 8 * (16 * (size_t)N + 8);
  }
  if (!c->hop_de) {
    CU(cudaMalloc(&c->hop_de, 8 * (size_t)N));
    c->bytes += 8 * (size_t)N;
    CU(cudaMemsetAsync(c->hop_de, 0, 8 * (size_t)N, c->stream));
  }
  int* cell_of = c->hop_cells;
  int* idx = cell_of + N;
  int* target = idx + N;
  int* count = target + N;
  int* start = count + kHopCellCap + 1;
  Lat l = c->lat;
  int treal = (int)(c->t % (unsigned long)c->tp);
  l.treal = treal;
  l.delx = c->p.edot * treal * c->p.dt;
  Cell cell = make_cell(l);
  double cr = 1.0, sr = 0.0;
  if (l.flow == BD_FLOW_EXT) {
    cr = l.cth;
    sr = l.sth;
  }
  double R = c->hop_R;
  HGeom g;
  for (int j = 0; j < 3; j++) {
    double a[3][3];
    for (int q = 0; q < 3; q++)
      for (int d = 0; d < 3; d++) a[q][d] = cell.H[d * 3 + q];
    const double* u = a[(j + 1) % 3];
    const double* v = a[(j + 2) % 3];
    double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2],
           cz = u[0] * v[1] - u[1] * v[0];
    int n = (int)floor(cell.V / sqrt(cx * cx + cy * cy + cz * cz) / R);
    g.n[j] = n >= 2 ? n - (n & 1) : 1;
  }
  while ((long)g.n[0] * g.n[1] * g.n[2] > kHopCellCap) {
    int d = g.n[0] >= g.n[1] && g.n[0] >= g.n[2] ? 0 : (g.n[1] >= g.n[2] ? 1 : 2);
    g.n[d] -= 2;
  }
  int ncell = g.n[0] * g.n[1] * g.n[2];
  // scratch (16 N + 8 doubles), in units of nch: [0, 4) the charges at their
  // sites at the colour's start, [4, 5) trial kinds (int), [5, 6) base
  // energies, [6, 7) charge values in track order, [8, 16) the accepted moves,
  // then the six entries of Q
  double4* cq = (double4*)c->hop_work;
  int* kind = (int*)(c->hop_work + 4 * (size_t)nch);
  double* de0 = c->hop_work + 5 * (size_t)nch;
  double* qk = c->hop_work + 6 * (size_t)nch;
  double4* moved = (double4*)(c->hop_work + 8 * (size_t)nch);
  c->launches += 5;
  k_charge_values<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->q, c->track, nch, qk);
  k_hop_cells<<<(nch + 255) / 256, 256, 0, c->stream>>>(cell, g, c->rx, c->ry, c->rz, c->track,
                                                        nch, cr, sr, cell_of, count);
  k_hop_scan<<<1, 1024, 0, c->stream>>>(ncell, count, start);
  k_hop_fill<<<(ncell + 3) / 4, 128, 0, c->stream>>>(cell_of, start, ncell, nch, idx);
  unsigned long long sweep = c->hop_sweeps++;
  k_hop_propose<<<nblk(nch, 8), 256, 0, c->stream>>>(
      l, c->rx, c->ry, c->rz, N, c->Nb, nch, c->track, c->nb_count, c->nb_rows, c->maxnb,
      c->p.philox_seed, sweep, target, kind);
  bool ewald = c->p.coulomb == BD_COULOMB_EWALD;
  HopEwald ew = {};
  int P = 0;
  if (ewald) {
    ew.cell = cell;
    ew.cr = cr;
    ew.sr = sr;
    ew.K = c->pmeK;
    ew.beta = c->cw_beta;
    ew.rc2 = c->cw_rc * c->cw_rc;
    ew.lambda_b = c->p.lambda_b;
    P = c->pme_p == 4 || c->pme_p == 6 ? c->pme_p : 8;
    double* Q6 = c->hop_work + 16 * (size_t)nch;
    int s;
    if ((s = coulomb_quadform(c, l, Q6)) != BD_OK) return s;
    ew.Q = Q6;
  }
  HGeom ccg = {};
  prof_begin(c, BD_PROF_HOP);
  for (int colour = 0; colour < 8; colour++) {
    // the charges at the colour's start and, with Ewald electrostatics, their
    // cell list and reciprocal potential
    c->launches += 3;
    k_gather_sites<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->rx, c->ry, c->rz, c->track, qk,
                                                             nch, cq);
    if (ewald) {
      int s;
      if ((s = coulomb_cells(c, l, cq, ccg.n, nullptr)) != BD_OK) return s;
      if ((s = coulomb_mesh_potential(c, l, cq)) != BD_OK) return s;
      ew.phi = c->cw_grid;
    }
#define HOP_COLOUR(P_)                                                                         \
  k_hop_base<P_><<<nblk(nch, 8), 256, 0, c->stream>>>(                                         \
      l, g, colour, c->rx, c->ry, c->rz, nch, idx, cell_of, c->track, qk, target, kind, cq,    \
      ccg, c->cw_start, c->cw_idx, (const double4*)c->cw_sorted, c->p.lambda_b, c->kappa_d,    \
      ew, de0);                                                                                \
  k_hop_accept<P_><<<ncell, 32, 0, c->stream>>>(                                               \
      l, g, colour, c->rx, c->ry, c->rz, start, idx, qk, target, kind, de0, c->track, c->old,  \
      c->cflags, moved, c->p.lambda_b, c->kappa_d, c->p.barrier, c->p.barrier2,                \
      c->p.philox_seed, sweep, c->hoplog, c->hop_de, ew)
    switch (P) {
      case 0: HOP_COLOUR(0); break;
      case 4: HOP_COLOUR(4); break;
      case 6: HOP_COLOUR(6); break;
      default: HOP_COLOUR(8);
    }
#undef HOP_COLOUR
  }
  prof_end(c, BD_PROF_HOP);
  c->launches += 2;
  k_clear_charges<<<(N + 255) / 256, 256, 0, c->stream>>>(c->cflags, c->q, N);
  k_scatter_charges<<<(nch + 255) / 256, 256, 0, c->stream>>>(c->track, qk, nch, c->cflags, c->q);
  return launch_ok(c);
}

}  // namespace bd

extern "C" int bd_download_hop_energies(bd_ctx* c, double* de) {
  if (!c || (c->nch > 0 && !de)) return BD_ERR_ARG;
  if (c->nch == 0) return BD_OK;
  if (!c->hop_de) return BD_ERR_STATE;
  CU(cudaMemcpyAsync(de, c->hop_de, 8 * (size_t)c->nch, cudaMemcpyDeviceToHost, c->stream));
  return check(c);
}
