// Real-space part of the particle-mesh mobility: pair lists, tensors, products.
//
// No counterpart in the reference (see bd_pme.cu).  The beads are taken four
// at a time (consecutive indices: neighbours along a chain, whose cutoff
// spheres nearly coincide).  A group's row lists every bead within the cutoff
// of one of its four, and per entry the four pair tensors T = t1 I + s w w^T,
// w = sqrt(|t2| / r^2) d, the sign s of t2 in the lowest mantissa bit of t1
// (zero where a pair is beyond the cutoff).  The product then reads a
// neighbour's input values once for four pairs, and positions and minimum
// images not at all.  The beads of a cell are in increasing index, so a row's
// order, and with it a product's rounding, is the same in every build.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "bd_real.cuh"

using namespace bd;

#define CU(call) BD_CU(call)

namespace {

constexpr int kGroup = 4;  // beads per row

// Real-space Beenakker kernel t1 I + t2 r r^T/r^2 (shear/src/main26.c:
// 1727-1741) at split parameter alpha; with FAR the r > 2 form at any r.  irr
// = 1/rr and ir = 1/r are formed once by the caller: a double division costs
// as much as ten multiplications, and the terms hold eight of them.
template <bool FAR>
__device__ __forceinline__ void real_kernel(double alpha, double rr, double r, double ir,
                                            double irr, double& t1, double& t2) {
  double a = alpha, a2 = a * a, a3 = a2 * a, a5 = a3 * a2, a7 = a5 * a2;
  double C1, C2, C3, C4;
  if (FAR || r > 2.0) {
    C1 = ir * (0.75 + 0.5 * irr);
    C2 = 4.0 * a7 * rr * rr + 3.0 * a3 * rr - 20.0 * a5 * rr - 4.5 * a + 14.0 * a3 + a * irr;
    C3 = ir * (0.75 - 1.5 * irr);
    C4 = -4.0 * a7 * rr * rr - 3.0 * a3 * rr + 16.0 * a5 * rr + 1.5 * a - 2.0 * a3 -
         3.0 * a * irr;
  } else {
    C1 = 1.0 - 0.28125 * r;
    C2 = 64.0 * a7 + 12.0 * a3 - 80.0 * a5 - 4.5 * a + 14.0 * a3 + 0.25 * a;
    C3 = 0.09375 * r;
    C4 = -64.0 * a7 - 12.0 * a3 + 64.0 * a5 + 1.5 * a - 2.0 * a3 - 0.75 * a;
  }
  const double irtpi = 0.56418958354775628695;  // 1/sqrt(pi)
  double ec = erfc(a * r), ex = exp(-a2 * rr) * irtpi;
  t1 = C1 * ec + C2 * ex;
  t2 = C3 * ec + C4 * ex;
}

// t1, t2 of the real-space pair tensor at split alpha, with calcHI's overlap
// convention for r < 2 (OVERLAP: the far form at alpha plus the overlap
// correction at its own split parameter alpha_ref).
template <bool OVERLAP>
__device__ __forceinline__ void pair_terms(double alpha, double alpha_ref, double rr, double r,
                                           double ir, double irr, double& t1, double& t2) {
  real_kernel<OVERLAP>(alpha, rr, r, ir, irr, t1, t2);
  if constexpr (OVERLAP) {
    double o1, o2, g1, g2;
    real_kernel<false>(alpha_ref, rr, r, ir, irr, o1, o2);
    real_kernel<true>(alpha_ref, rr, r, ir, irr, g1, g2);
    t1 += o1 - g1;
    t2 += o2 - g2;
  }
}

// Cells of the real-space list (fractional, width >= rc).
struct RGeom {
  int n[3];
};

__global__ void k_rl_count(Cell cell, RGeom g, const double* __restrict__ rx,
                           const double* __restrict__ ry, const double* __restrict__ rz,
                           double cr, double sr, int N, int* cell_of, int* cell_count) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int cd[3];
  double x = rx[i] * cr - ry[i] * sr, y = rx[i] * sr + ry[i] * cr;
  int c = cell_of_pos(cell, g.n, x, y, rz[i], cd);
  cell_of[i] = c;
  atomicAdd(&cell_count[c], 1);
}

__global__ void k_rl_scan(int ncell, int* cell_count, int* cell_start, int* cursor) {
  __shared__ int part[1024];
  int t = threadIdx.x, nt = blockDim.x;
  int per = (ncell + nt - 1) / nt, lo = t * per, hi = min(ncell, lo + per), s = 0;
  for (int c = lo; c < hi; c++) s += cell_count[c];
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
    cell_start[c] = b;
    cursor[c] = 0;
    b += cell_count[c];
    cell_count[c] = 0;
  }
  if (t == nt - 1) cell_start[ncell] = part[t];
}

__global__ void k_rl_fill(const int* __restrict__ cell_of, const int* __restrict__ cell_start,
                          int* cursor, int* beads, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int c = cell_of[i];
  beads[cell_start[c] + atomicAdd(&cursor[c], 1)] = i;
}

// Positions in cell order, a cell's beads in increasing index, the index in the
// fourth component: the row build streams a cell's beads with one contiguous
// load each.  One block per cell, each bead placed by its rank.
__global__ void __launch_bounds__(256) k_rl_order(const int* __restrict__ cell_start,
                                                  const int* __restrict__ beads,
                                                  const double4* __restrict__ pos,
                                                  double4* spos) {
  __shared__ int s[1024];
  const int lo = cell_start[blockIdx.x], n = cell_start[blockIdx.x + 1] - lo;
  for (int e0 = 0; e0 < n; e0 += blockDim.x) {
    const int e = e0 + threadIdx.x, v = e < n ? beads[lo + e] : 0;
    int rank = 0;
    for (int t0 = 0; t0 < n; t0 += 1024) {
      const int m = min(1024, n - t0);
      __syncthreads();
      for (int q = threadIdx.x; q < m; q += blockDim.x) s[q] = beads[lo + t0 + q];
      __syncthreads();
      if (e < n)
        for (int q = 0; q < m; q++) rank += s[q] < v;
    }
    if (e < n) {
      double4 p = pos[v];
      p.w = __longlong_as_double((long long)v);
      spos[lo + rank] = p;
    }
  }
}

// t1 with the sign of t2 in its lowest mantissa bit.
__device__ __forceinline__ float with_sign(float, double t1, double t2) {
  return __uint_as_float((__float_as_uint((float)t1) & ~1u) | (t2 < 0.0 ? 1u : 0u));
}
__device__ __forceinline__ double with_sign(double, double t1, double t2) {
  return __longlong_as_double((__double_as_longlong(t1) & ~1ll) | (t2 < 0.0 ? 1ll : 0ll));
}

// The four tensors of an entry: 16 numbers, for beads (0, 1) and (2, 3) the
// pairs of t1, w_x, w_y, w_z, so that the product takes two beads per
// instruction.
template <typename R>
__device__ __forceinline__ void store_tensor(R* entry, int b, double t1, double t2, double sw,
                                             double dx, double dy, double dz) {
  R* o = entry + 8 * (b >> 1) + (b & 1);
  o[0] = with_sign((R)0, t1, t2);
  o[2] = (R)(sw * dx);
  o[4] = (R)(sw * dy);
  o[6] = (R)(sw * dz);
}

// Neighbour indices of the groups' rows, cap entries a row, in no order.  One
// warp per group.  For each of its beads the at most 27 neighbour cells form
// one candidate list; the lanes test 32 candidates at a time and queue the
// hits in shared memory.  Batches of hits are then tested against the group's
// earlier beads: a neighbour is listed by the first bead that has it within
// the cutoff.  Bound by the FP64 pipe: 193 M candidates at 50 000 beads, cutoff
// 14.5, 0.86 ms (a thread per bead forming rows and tensors together took 6.0, a
// warp per bead 1.3; this and k_rl_tensors 1.5, for rows the product reads 1.7 times
// faster).
__global__ void __launch_bounds__(128, 4)
    k_rl_find(Cell cell, RGeom g, const double4* __restrict__ pos, int N, int ngroup,
              const int* __restrict__ cell_start, const double4* __restrict__ spos, double rc2,
              int cap, int* cnt, int* rows, int* need, int* err) {
  __shared__ CandList c_list[4];
  __shared__ int c_queue[4][64];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * 4 + wl;
  if (grp >= ngroup) return;
  const int i0 = kGroup * grp, nb = min(kGroup, N - i0);
  const Image image(cell);
  int* row = rows + (size_t)grp * cap;
  int* queue = c_queue[wl];
  int n = 0, nq = 0;
  // the first m hits of bead b: those that no earlier bead lists
  auto list = [&](int b, int m) {
    bool keep = lane < m;
    int j = 0;
    if (keep) {
      const double4 pj = spos[queue[lane]];
      j = (int)__double_as_longlong(pj.w);
      for (int q = 0; q < b; q++) {
        double dx, dy, dz;
        if (j != i0 + q && !(image(pj, pos[i0 + q], dx, dy, dz) >= rc2)) keep = false;
      }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, keep);
    const int at = n + __popc(hit & ((1u << lane) - 1u));
    if (keep && at < cap) row[at] = j;
    n += __popc(hit);
    nq -= m;
    const int rest = lane < nq ? queue[m + lane] : 0;
    __syncwarp();
    if (lane < nq) queue[lane] = rest;
    __syncwarp();
  };
#pragma unroll 1
  for (int b = 0; b < nb; b++) {
    const double4 pb = pos[i0 + b];
    int cd[3], cl = 0, next_at = -1;
    cell_of_pos(cell, g.n, pb.x, pb.y, pb.z, cd);
    const int total = c_list[wl].open(g.n, cd, cell_start);
    // the next candidate's load is in flight while this one is tested
    double4 next = pb;
    auto fetch = [&](int m) {
      next_at = -1;
      if (m < total) {
        next_at = c_list[wl].at(m, cl);
        next = spos[next_at];
      }
    };
    fetch(lane);
#pragma unroll 1
    for (int m0 = 0; m0 < total; m0 += 32) {
      const int at = next_at;
      const double4 pj = next;
      fetch(m0 + 32 + lane);
      double dx, dy, dz;
      const double rr = image(pj, pb, dx, dy, dz);
      const bool in = at >= 0 && !(rr >= rc2) && (int)__double_as_longlong(pj.w) != i0 + b;
      const unsigned hit = __ballot_sync(0xffffffffu, in);
      if (in) queue[nq + __popc(hit & ((1u << lane) - 1u))] = at;
      nq += __popc(hit);
      __syncwarp();
      if (nq >= 32) list(b, 32);
    }
    if (nq > 0) list(b, nq);
  }
  if (lane == 0) {
    cnt[grp] = min(n, cap);
    if (n > cap) {
      if (need)
        atomicMax(need, n);  // the host grows the rows and builds them again
      else
        atomicOr(err, ERRB_NBR_OVERFLOW);
    }
  }
}

// The four tensors of every entry, a warp per group, and each bead's number of
// pairs against an explicit cap.  Entry k at rw[16 (group cap + k)].  32 entries
// at a time are formed in shared memory and written side by side (from the
// lanes, 64 bytes apart, every sector would be written eight times).
// Overlapping pairs (r < 2), whose terms cost three times as much, are queued
// and formed 32 at a time.  Bound by the FP64 pipe (erfc, exp): 0.62 ms at
// 50 000 beads, cutoff 14.5; 0.76 with each lane writing its own entry.
template <typename R>
__global__ void __launch_bounds__(128, 4)
    k_rl_tensors(Cell cell, const double4* __restrict__ pos, int N, int ngroup,
                 const int* __restrict__ cnt, const int* __restrict__ rows, int cap, double rc2,
                 double alpha, double alpha_ref, int bead_cap, R* rw, int* err) {
  __shared__ int c_queue[4][160];  // 4 k + b of overlapping pairs
  __shared__ alignas(16) R s_entry[4][32 * 20];  // entries 20 apart: fewer bank conflicts
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * 4 + wl;
  if (grp >= ngroup) return;
  const int i0 = kGroup * grp, nb = min(kGroup, N - i0), n = cnt[grp];
  const Image image(cell);
  const int* row = rows + (size_t)grp * cap;
  R* out = rw + 16 * (size_t)grp * cap;
  int* queue = c_queue[wl];
  int nq = 0, count[kGroup] = {0, 0, 0, 0};
  auto form = [&](auto overlap, R* entry, int b, double rr, double dx, double dy, double dz) {
    constexpr bool OV = decltype(overlap)::value;
    const double r = sqrt(rr), ir = 1.0 / r, irr = ir * ir;
    double t1, t2;
    pair_terms<OV>(alpha, alpha_ref, rr, r, ir, irr, t1, t2);
    store_tensor(entry, b, t1, t2, sqrt(fabs(t2)) * ir, dx, dy, dz);
  };
  auto flush = [&](int m) {
    if (lane < m) {
      const int k = queue[nq - m + lane] >> 2, b = queue[nq - m + lane] & 3;
      double dx, dy, dz;
      const double rr = image(pos[row[k]], pos[i0 + b], dx, dy, dz);
      form(std::integral_constant<bool, true>(), out + 16 * (size_t)k, b, rr, dx, dy, dz);
    }
    nq -= m;
    __syncwarp();
  };
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += 32) {
    const int k = k0 + lane, m = min(32, n - k0);
    R* entry = s_entry[wl] + 20 * lane;
    const int j = k < n ? row[k] : 0;
    const double4 pj = pos[j];
#pragma unroll 1
    for (int b = 0; b < kGroup; b++) {
      bool near = false;
      double dx, dy, dz;
      const double rr = image(pj, pos[min(i0 + b, N - 1)], dx, dy, dz);
      if (k < n && b < nb && j != i0 + b && !(rr >= rc2)) {
        count[0] += b == 0, count[1] += b == 1, count[2] += b == 2, count[3] += b == 3;
        near = rr < 4.0;
        if (!near) form(std::integral_constant<bool, false>(), entry, b, rr, dx, dy, dz);
      } else {
        store_tensor(entry, b, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
      }
      const unsigned hit = __ballot_sync(0xffffffffu, near);
      if (near) queue[nq + __popc(hit & ((1u << lane) - 1u))] = 4 * k + b;
      nq += __popc(hit);
    }
    __syncwarp();
    constexpr int WORDS = (int)sizeof(R);  // 16-byte words an entry
    float4* to = (float4*)(out + 16 * (size_t)k0);
    for (int e = lane; e < m * WORDS; e += 32)
      to[e] = ((const float4*)(s_entry[wl] + 20 * (e / WORDS)))[e % WORDS];
    __syncwarp();
    while (nq >= 32) flush(32);
  }
  if (nq > 0) flush(nq);
  int longest = 0;
#pragma unroll
  for (int b = 0; b < kGroup; b++) {
    for (int o = 16; o > 0; o >>= 1) count[b] += __shfl_xor_sync(0xffffffffu, count[b], o);
    longest = max(longest, count[b]);
  }
  if (lane == 0 && bead_cap > 0 && longest > bead_cap) atomicOr(err, ERRB_NBR_OVERFLOW);
}

// ---------------------------------------------------------------------------

// Two beads at a time: the beads' numbers in the halves, one input value for both.
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }
__device__ __forceinline__ double twice(double x) { return x; }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d, x = *reinterpret_cast<unsigned long long*>(&a),
                        y = *reinterpret_cast<unsigned long long*>(&b);
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d, x = *reinterpret_cast<unsigned long long*>(&a),
                        y = *reinterpret_cast<unsigned long long*>(&b),
                        z = *reinterpret_cast<unsigned long long*>(&c);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ double2 mul2(double2 a, double b) {
  return make_double2(a.x * b, a.y * b);
}
__device__ __forceinline__ double2 fma2(double2 a, double b, double2 c) {
  return make_double2(fma(a.x, b, c.x), fma(a.y, b, c.y));
}
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
// negative where the bead's t1 carries a negative sign
__device__ __forceinline__ float2 signed_by(float2 t1, float2 a) {
  return make_float2(__uint_as_float(__float_as_uint(a.x) ^ (__float_as_uint(t1.x) << 31)),
                     __uint_as_float(__float_as_uint(a.y) ^ (__float_as_uint(t1.y) << 31)));
}
__device__ __forceinline__ double2 signed_by(double2 t1, double2 a) {
  return make_double2(__double_as_longlong(t1.x) & 1 ? -a.x : a.x,
                      __double_as_longlong(t1.y) & 1 ? -a.y : a.y);
}

template <typename R>
struct Real2;
template <>
struct Real2<float> {
  using T = float2;
};
template <>
struct Real2<double> {
  using T = double2;
};

__device__ __forceinline__ void copy_async(void* to, const void* from, int bytes16) {
  unsigned d = (unsigned)__cvta_generic_to_shared(to);
  if (bytes16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// The real-space sums of NP packed pairs (p0 on) and the rest of the product.
// One warp per group of four beads: a lane serves one pair and every S-th
// entry of the row (S = 32 / NP), so NP lanes read a neighbour's packed values
// (component c of pair p at vpk[(c N + j) np + p]) side by side and use them
// for the four beads, two at a time.  The row (68 bytes an entry, read once)
// streams through shared memory, about 30 entries at a time with two more such pieces under
// way: with loads to registers, an entry ahead, too few bytes were in flight
// to cover the latency of L2 and HBM (430 us at 50 000 beads, cutoff 14.5,
// five pairs).  FP32: partial sums of about 16 entries folded into a second
// set; lanes added in FP64.  Five pairs: 257 us at 50 000 beads, cutoff 14.5
// (a warp per bead, every neighbour's values read once per bead: 435); at 8000
// beads, cutoff 12.1, 38 us by one warp a group against 50.
// SPLIT warps share a group's row.
template <int NP, typename R>
struct Stage {
  static constexpr int S = 32 / NP, ITS = 32 / S, CH = S * ITS;  // entries a piece
  alignas(16) R w[16 * CH];
  int j[(CH + 3) / 4 * 4];
};

template <int NP, int SPLIT, typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 4 : 2)
    k_real_apply(const int* __restrict__ cnt, const int* __restrict__ rows,
                 const R* __restrict__ rw, int cap,
                 const typename Real2<R>::T* __restrict__ vpk, int np, int p0, int N, int ngroup,
                 Finish fin) {
  using V = typename Real2<R>::T;
  using P = Stage<NP, R>;
  constexpr int S = P::S, ITS = P::ITS, CH = P::CH, DEEP = sizeof(R) == 4 ? 3 : 2, W = 25;
  constexpr int FOLD = 16 / ITS, PER = (int)sizeof(R);  // 16-byte words an entry
  union Shared {
    P stage[4][DEEP];
    R sum[4][32 * W];
  };
  __shared__ __align__(16) unsigned char raw[sizeof(Shared)];
  Shared& sh = *reinterpret_cast<Shared*>(raw);
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * (4 / SPLIT) + wl / SPLIT, piece0 = wl % SPLIT;
  const int slot = lane / NP, pr = lane % NP;  // slot S and up: idle lanes
  V sum[2][6], part[2][6];  // beads (0, 1), (2, 3); values 3 h + c
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int e = 0; e < 6; e++) sum[b][e].x = sum[b][e].y = part[b][e].x = part[b][e].y = 0;
  if (grp < ngroup) {
    const int n = cnt[grp];
    const int* row = rows + (size_t)grp * cap;
    const R* rq = rw + 16 * (size_t)grp * cap;
    const V* vp = vpk + p0 + pr;
    const size_t plane = (size_t)N * np;
    P* st = sh.stage[wl];
    auto issue = [&](int piece, int buf) {
      const int k0 = piece * CH, m = min(CH, n - k0);
      const char* from = (const char*)(rq + 16 * (size_t)k0);
      for (int e = lane; e < m * PER; e += 32)
        copy_async((char*)st[buf].w + 16 * e, from + 16 * e, 1);
      if (lane < m) copy_async(st[buf].j + lane, row + k0 + lane, 0);
      copy_commit();
    };
#pragma unroll
    for (int d = 0; d < DEEP - 1; d++) issue(piece0 + d * SPLIT, d);
    int buf = 0, folded = 0;
#pragma unroll 1
    for (int piece = piece0; piece * CH < n; piece += SPLIT) {
      copy_wait<DEEP - 2>();
      __syncwarp();
      const int m = min(CH, n - piece * CH);
      const P& p = st[buf];
      V x[ITS][3];
#pragma unroll
      for (int t = 0; t < ITS; t++) {
        const int k = t * S + slot;
        const V* vj = vp + (size_t)(slot < S && k < m ? p.j[k] : 0) * np;
#pragma unroll
        for (int c = 0; c < 3; c++) x[t][c] = __ldg(vj + c * plane);
      }
      // the buffer used last is free: every lane is past the barrier above
      issue(piece + (DEEP - 1) * SPLIT, buf == 0 ? DEEP - 1 : buf - 1);
#pragma unroll
      for (int t = 0; t < ITS; t++) {
        const int k = t * S + slot;
        if (slot < S && k < m) {
#pragma unroll
          for (int b = 0; b < 2; b++) {
            V t1, w0, w1, w2;
            if constexpr (sizeof(R) == 4) {
              const float4 u = *(const float4*)(p.w + 16 * k + 8 * b),
                           v = *(const float4*)(p.w + 16 * k + 8 * b + 4);
              t1 = make_float2(u.x, u.y), w0 = make_float2(u.z, u.w);
              w1 = make_float2(v.x, v.y), w2 = make_float2(v.z, v.w);
            } else {
              const V* q = (const V*)(p.w + 16 * k + 8 * b);
              t1 = q[0], w0 = q[1], w1 = q[2], w2 = q[3];
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const auto y0 = twice(h ? x[t][0].y : x[t][0].x),
                         y1 = twice(h ? x[t][1].y : x[t][1].x),
                         y2 = twice(h ? x[t][2].y : x[t][2].x);
              const V d = signed_by(t1, fma2(w2, y2, fma2(w1, y1, mul2(w0, y0))));
              V* o = part[b] + 3 * h;
              o[0] = fma2(w0, d, fma2(t1, y0, o[0]));
              o[1] = fma2(w1, d, fma2(t1, y1, o[1]));
              o[2] = fma2(w2, d, fma2(t1, y2, o[2]));
            }
          }
        }
      }
      buf = buf + 1 == DEEP ? 0 : buf + 1;
      if (++folded == FOLD) {
        folded = 0;
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
          for (int e = 0; e < 6; e++) {
            sum[b][e].x += part[b][e].x;
            sum[b][e].y += part[b][e].y;
            part[b][e].x = part[b][e].y = 0;
          }
      }
    }
    copy_wait<0>();
  }
  __syncthreads();  // the stages' memory holds the sums from here on
  R* o = sh.sum[wl] + lane * W;
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int e = 0; e < 6; e++) {
      o[12 * b + e] = sum[b][e].x + part[b][e].x;
      o[12 * b + 6 + e] = sum[b][e].y + part[b][e].y;
    }
  __syncthreads();
  if (grp >= ngroup) return;
  const int w0 = wl / SPLIT * SPLIT;
  for (int e = lane + 32 * piece0; e < 6 * kGroup * NP; e += 32 * SPLIT) {
    const int b = e / (6 * NP), p = e / 6 % NP, i = kGroup * grp + b;
    if (i >= N) break;
    double s = 0;
    for (int w = w0; w < w0 + SPLIT; w++)
      for (int u = 0; u < S; u++) s += (double)sh.sum[w][(u * NP + p) * W + 6 * b + e % 6];
    fin.write(s, p0 + p, e % 6, i);
  }
}

template <int NP, typename R>
void launch_apply(bd_ctx* c, int np, int p0, const Finish& fin) {
  const int ng = (c->N + kGroup - 1) / kGroup;
#define REAL(SPLIT_)                                                                      \
  k_real_apply<NP, SPLIT_, R><<<nblk(ng, 4 / SPLIT_), 128, 0, c->stream>>>(               \
      c->rl_cnt, c->rl_rows, (const R*)c->rl_w, c->rl_cap,                                \
      (const typename Real2<R>::T*)c->pme_vpk, np, p0, c->N, ng, fin)
  // More warps a group fill the chip sooner, fewer start fewer pieces.  By four,
  // two and one, five pairs FP32: 500 beads 6.1, 8.0, 12.6 us, 8000 41.8, 46.5, 63.7,
  // 16 000 70, 74, 79; FP64 8000 85, 90, 107, 16 000 151, 147, 160; one pair FP32
  // 8000 24.0, 20.9, 24.4, 16 000 45.5, 35.2, 34.5.  At 50 000 beads of a run's
  // chains five pairs took 268 by four and 257 by one, one pair 118 by two and 114
  // by one.
  const int four = NP < 5 ? 148 * 12 : sizeof(R) == 8 ? 148 * 20 : 148 * 40;
  if (ng >= 148 * 40)
    REAL(1);
  else if (ng < four)
    REAL(4);
  else
    REAL(2);
#undef REAL
}

template <typename R>
int apply_t(bd_ctx* c, int np, const Finish& fin) {
  for (int p0 = 0; p0 < np; p0 += 5) {
    c->launches++;
    switch (std::min(5, np - p0)) {
      case 1: launch_apply<1, R>(c, np, p0, fin); break;
      case 2: launch_apply<2, R>(c, np, p0, fin); break;
      case 3: launch_apply<3, R>(c, np, p0, fin); break;
      case 4: launch_apply<4, R>(c, np, p0, fin); break;
      default: launch_apply<5, R>(c, np, p0, fin);
    }
  }
  return launch_ok(c);
}

}  // namespace

namespace bd {

// Rows of cap entries for every group; without memory for them there are none
// (rl_rows null) and the mobility is not built.
static int rows_alloc(bd_ctx* c, int cap) {
  size_t ng = ((size_t)c->N + kGroup - 1) / kGroup, es = c->pme_f32 ? 4 : 8;
  size_t old = (size_t)c->rl_cap, each = 4 + 4 * es * kGroup;
  if (c->rl_rows) {
    CU(cudaStreamSynchronize(c->stream));
    free_all({&c->rl_rows, &c->rl_w});
    c->bytes -= each * ng * old;
  }
  c->rl_cap = 0;
  int s = alloc_all(c, {{&c->rl_rows, 4 * ng * cap}, {&c->rl_w, 4 * es * kGroup * ng * cap}});
  if (s == BD_OK) c->rl_cap = cap;
  return s;
}

// Rows before any have overflowed: an explicit cap per bead bounds a group's
// row by four times that; the default is 2.5 times the mean number of beads
// within the cutoff at the system's density, at least 512 (rows that overflow
// it are grown); no row is longer than N.
static int first_cap(const bd_ctx* c) {
  long cap;
  if (c->p.pme_max_pairs > 0) {
    cap = (long)kGroup * c->p.pme_max_pairs;
  } else {
    double mean = 4.0 / 3.0 * M_PI * c->pme_rc * c->pme_rc * c->pme_rc * c->N / c->boxvol;
    cap = std::max(512, ((int)ceil(2.5 * mean) + 31) / 32 * 32);
  }
  return (int)std::min(cap, (long)std::max(c->N, 1));
}

int real_alloc(bd_ctx* c) {
  const size_t N = c->N;
  c->rl_ncell_cap = 4096;
  int s = alloc_all(c, {{&c->rl_cnt, 4 * N},
                        {&c->rl_need, 4},
                        {&c->rl_cell_of, 4 * N},
                        {&c->rl_spos, 32 * N},
                        {&c->rl_beads, 4 * N},
                        {&c->rl_cell_count, 4 * (size_t)c->rl_ncell_cap},
                        {&c->rl_cell_start, 4 * (size_t)(c->rl_ncell_cap + 1)},
                        {&c->rl_cursor, 4 * (size_t)c->rl_ncell_cap}});
  if (s != BD_OK) return s;
  CU(cudaMemsetAsync(c->rl_need, 0, 4, c->stream));
  CU(cudaMemsetAsync(c->rl_cell_count, 0, 4 * (size_t)c->rl_ncell_cap, c->stream));
  return BD_OK;
}

void real_free(bd_ctx* c) {
  free_all({&c->rl_rows, &c->rl_w, &c->rl_cnt, &c->rl_need, &c->rl_cell_of, &c->rl_spos,
            &c->rl_beads, &c->rl_cell_count, &c->rl_cell_start, &c->rl_cursor});
  c->rl_cap = 0;
}

// The groups' rows for the positions in rl_pos (lab frame; rx, ry, rz and the
// rotation (cr, sr) give the same); alpha_ref is calcHI's split parameter.
int real_prepare(bd_ctx* c, const Cell& cell, double cr, double sr, double alpha_ref) {
  int s, N = c->N;
  double rc = c->pme_rc, alpha = c->pme_alpha;
  if (!c->rl_rows && (s = rows_alloc(c, first_cap(c))) != BD_OK) return s;
  // real-space cells: perpendicular widths V/|a_j x a_k|
  double w[3];
  {
    const double* H = cell.H;
    double a[3][3];
    for (int j = 0; j < 3; j++)
      for (int d = 0; d < 3; d++) a[j][d] = H[d * 3 + j];
    for (int j = 0; j < 3; j++) {
      const double* u = a[(j + 1) % 3];
      const double* v = a[(j + 2) % 3];
      double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2],
             cz = u[0] * v[1] - u[1] * v[0];
      w[j] = cell.V / sqrt(cx * cx + cy * cy + cz * cz);
    }
  }
  if (2 * rc > std::min(w[0], std::min(w[1], w[2]))) return BD_ERR_ARG;  // rc beyond half a width
  RGeom g;
  for (int d = 0; d < 3; d++) g.n[d] = std::max(1, (int)floor(w[d] / rc));
  while ((long)g.n[0] * g.n[1] * g.n[2] > c->rl_ncell_cap) {
    int d = g.n[0] >= g.n[1] && g.n[0] >= g.n[2] ? 0 : (g.n[1] >= g.n[2] ? 1 : 2);
    g.n[d]--;
  }
  int ncell = g.n[0] * g.n[1] * g.n[2];
  c->launches += 4;
  k_rl_count<<<nblk(N, 256), 256, 0, c->stream>>>(cell, g, c->rx, c->ry, c->rz, cr, sr, N,
                                                  c->rl_cell_of, c->rl_cell_count);
  k_rl_scan<<<1, 1024, 0, c->stream>>>(ncell, c->rl_cell_count, c->rl_cell_start, c->rl_cursor);
  k_rl_fill<<<nblk(N, 256), 256, 0, c->stream>>>(c->rl_cell_of, c->rl_cell_start, c->rl_cursor,
                                                 c->rl_beads, N);
  c->launches++;
  k_rl_order<<<ncell, 256, 0, c->stream>>>(c->rl_cell_start, c->rl_beads,
                                           (const double4*)c->rl_pos, (double4*)c->rl_spos);
  if ((s = launch_ok(c)) != BD_OK) return s;
  // the rows; with the default cap (no pme_max_pairs), rows that
  // overflow it are grown to 1.25 times the longest row and built again
  int* need = c->p.pme_max_pairs > 0 ? nullptr : c->rl_need;
  const int ng = (N + kGroup - 1) / kGroup;
  for (int pass = 0; pass < 2; pass++) {
    c->launches++;
    k_rl_find<<<nblk(ng, 4), 128, 0, c->stream>>>(
        cell, g, (const double4*)c->rl_pos, N, ng, c->rl_cell_start, (const double4*)c->rl_spos,
        rc * rc, c->rl_cap, c->rl_cnt, c->rl_rows, need, c->err);
    if (!need) break;
    int longest = 0;
    CU(cudaMemcpyAsync(&longest, need, 4, cudaMemcpyDeviceToHost, c->stream));
    if ((s = check(c)) != BD_OK) return s;
    if (longest <= c->rl_cap) break;
    CU(cudaMemsetAsync(c->rl_need, 0, 4, c->stream));
    if ((s = rows_alloc(c, std::min(N, ((int)ceil(1.25 * longest) + 31) / 32 * 32))) != BD_OK)
      return s;
  }
  c->launches++;
  if (c->pme_f32)
    k_rl_tensors<float><<<nblk(ng, 4), 128, 0, c->stream>>>(
        cell, (const double4*)c->rl_pos, N, ng, c->rl_cnt, c->rl_rows, c->rl_cap, rc * rc, alpha,
        alpha_ref, c->p.pme_max_pairs, (float*)c->rl_w, c->err);
  else
    k_rl_tensors<double><<<nblk(ng, 4), 128, 0, c->stream>>>(
        cell, (const double4*)c->rl_pos, N, ng, c->rl_cnt, c->rl_rows, c->rl_cap, rc * rc, alpha,
        alpha_ref, c->p.pme_max_pairs, (double*)c->rl_w, c->err);
  return launch_ok(c);
}

int real_apply(bd_ctx* c, int np, const Finish& fin) {
  return c->pme_f32 ? apply_t<float>(c, np, fin) : apply_t<double>(c, np, fin);
}

}  // namespace bd
