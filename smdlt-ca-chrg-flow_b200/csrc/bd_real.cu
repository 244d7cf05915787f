// Real-space part of the particle-mesh mobility: pair lists, tensors, products.
//
// No counterpart in the reference (see bd_pme.cu).  The beads are taken four
// at a time, neighbours whose cutoff spheres nearly coincide: consecutive indices
// along a chain, or neighbours in space where chains are short (by_index).  A
// group's row lists every bead within the cutoff
// of one of its four, and per entry the four pair tensors (zero where a pair is
// beyond the cutoff), so that a product reads a neighbour once for four pairs.
// Two forms:
//  * whole tensors, in FP32 contexts with noise blocks: T = t1 I + s w w^T, w =
//    sqrt(|t2| / r^2) d, the sign s of t2 in the lowest mantissa bit of t1.  64
//    bytes an entry; positions and minimum images are not needed, and up to five
//    pairs of right-hand sides share the reading (k_real_apply, FP32 sums);
//  * t1 and t2 / r^2 in FP64 contexts and in FP32 ones with one right-hand side:
//    64 and 32 bytes an entry, the displacements from the frozen FP64 positions,
//    FP64 inputs and sums (k_real_sum).  Whole FP64 tensors are twice the bytes
//    and give up a bit of t1: a single FP64 product of 50 000 beads (cutoff 14.5)
//    took 580 us with them, 392 so; of 8000 (12.1) 143 and 114; five pairs of 8000
//    333 and 331.
// The beads of a cell are in increasing index, so a row's order, and with it a
// product's rounding, is the same in every build.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "bd_real.cuh"

using namespace bd;

#define CU(call) BD_CU(call)

namespace {

constexpr int kGroup = 4;  // beads per row

// Whether groups are consecutive indices: chains of a multiple of four beads fill
// whole groups, of long ones few groups straddle two.  The others go by small
// cells: products of 50 000 beads (cutoff 14.5) by index and by cells, single FP32,
// single FP64 and ten FP32, monomers 558, 759, 1367 and 319, 452, 931 us; chains of
// 5 333, 448, 1009 and 294, 406, 916; of 8 286, 392, 892 and 292, 404, 913; of 10
// 308, 423, 963 and 290, 402, 918; of 25 304, 420, 958 and 300, 413, 941, for which
// the build takes 1.90 and 2.04 ms.
inline bool by_index(int Nb) { return Nb % kGroup == 0 || Nb >= 16; }

// Bead of a place in the groups' order: gpos holds the beads' positions in that
// order, the index in the fourth component.
__device__ __forceinline__ int bead_of(const double4& p) {
  return (int)__double_as_longlong(p.w);
}

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

// Positions in cell order, a cell's beads in increasing index: the row build streams a cell's beads with one contiguous
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
    if (e < n) spos[lo + rank] = pos[v];
  }
}

// Positions in the order of the cells, a cell's beads in increasing index: the
// groups' order of unchained beads.  One warp per cell of a bead or two.
__global__ void __launch_bounds__(256) k_rl_group(const int* __restrict__ cell_start, int ncell,
                                                  const int* __restrict__ beads,
                                                  const double4* __restrict__ pos, double4* gpos) {
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= ncell) return;
  const int lo = cell_start[c], n = cell_start[c + 1] - lo;
  for (int e = lane; e < n; e += 32) {
    const int v = beads[lo + e];
    int rank = 0;
    for (int q = 0; q < n; q++) rank += beads[lo + q] < v;
    gpos[lo + rank] = pos[v];
  }
}

// t1 with the sign of t2 in its lowest mantissa bit.
__device__ __forceinline__ float with_sign(double t1, double t2) {
  return __uint_as_float((__float_as_uint((float)t1) & ~1u) | (t2 < 0.0 ? 1u : 0u));
}

// The four tensors of an entry: 16 numbers, for beads (0, 1) and (2, 3) the
// pairs of t1, w_x, w_y, w_z, so that the product takes two beads per
// instruction.
__device__ __forceinline__ void store_tensor(float* entry, int b, double t1, double t2, double sw,
                                             double dx, double dy, double dz) {
  float* o = entry + 8 * (b >> 1) + (b & 1);
  o[0] = with_sign(t1, t2);
  o[2] = (float)(sw * dx);
  o[4] = (float)(sw * dy);
  o[6] = (float)(sw * dz);
}

// Place of bead b's pair in entry k of a row of (t1, t2 / r^2): 32 entries of
// each bead side by side.
__device__ __forceinline__ size_t pair_at(int k, int b) {
  return ((size_t)(k >> 5) * kGroup + b) * 32 + (k & 31);
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
    k_rl_find(Cell cell, RGeom g, const double4* __restrict__ gpos, int N, int ngroup,
              const int* __restrict__ cell_start, const double4* __restrict__ spos, double rc2,
              int cap, int* cnt, int* rows, int* need, int* err) {
  __shared__ CandList c_list[4];
  __shared__ int c_queue[4][64];
  __shared__ double4 s_group[4][kGroup];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * 4 + wl;
  if (grp >= ngroup) return;
  const int i0 = kGroup * grp, nb = min(kGroup, N - i0);
  const Image image(cell);
  int* row = rows + (size_t)grp * cap;
  int* queue = c_queue[wl];
  const double4* group = s_group[wl];
  if (lane < nb) s_group[wl][lane] = gpos[i0 + lane];
  __syncwarp();
  int n = 0, nq = 0;
  // the first m hits of bead b: those that no earlier bead lists
  auto list = [&](int b, int m) {
    bool keep = lane < m;
    int j = 0;
    if (keep) {
      const double4 pj = spos[queue[lane]];
      j = bead_of(pj);
      for (int q = 0; q < b; q++) {
        const double4 pq = group[q];
        double dx, dy, dz;
        if (j != bead_of(pq) && !(image(pj, pq, dx, dy, dz) >= rc2)) keep = false;
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
    const double4 pb = group[b];
    const int own = bead_of(pb);
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
      const bool in = at >= 0 && !(rr >= rc2) && bead_of(pj) != own;
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

// The pair tensors of every entry, a warp per group, and each bead's number of
// pairs against an explicit cap.  WHOLE: 16 numbers an entry at rw[16 (group cap
// + k)]; 32 entries at a time are formed in shared memory and written side by
// side (from the lanes, 64 bytes apart, every sector would be written eight
// times).  Else (t1, t2 / r^2) at pair_at.  Overlapping pairs (r < 2), whose
// terms cost three times as much, are queued and formed 32 at a time.  Bound by
// the FP64 pipe (erfc, exp): 0.62 ms at 50 000 beads, cutoff 14.5; 0.76 with each
// lane writing its own entry.
template <typename R, bool WHOLE>
__global__ void __launch_bounds__(128, 4)
    k_rl_tensors(Cell cell, const double4* __restrict__ pos, const double4* __restrict__ gpos,
                 int N, int ngroup,
                 const int* __restrict__ cnt, const int* __restrict__ rows, int cap, double rc2,
                 double alpha, double alpha_ref, int bead_cap, void* rw, int* err) {
  using T2 = typename Real2<R>::T;
  __shared__ int c_queue[4][160];  // 4 k + b of overlapping pairs
  // entries 20 numbers apart: fewer bank conflicts
  __shared__ alignas(16) float s_entry[WHOLE ? 4 : 1][WHOLE ? 32 * 20 : 4];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * 4 + wl;
  if (grp >= ngroup) return;
  const int i0 = kGroup * grp, nb = min(kGroup, N - i0), n = cnt[grp];
  const Image image(cell);
  const int* row = rows + (size_t)grp * cap;
  float* whole = (float*)rw + 16 * (size_t)grp * cap;
  T2* out = (T2*)rw + kGroup * (size_t)grp * cap;
  int* queue = c_queue[wl];
  int nq = 0, count[kGroup] = {0, 0, 0, 0};
  // pair (k, b): to entry (WHOLE) or to its place
  auto form = [&](auto overlap, float* entry, int k, int b, double rr, double dx, double dy,
                  double dz) {
    constexpr bool OV = decltype(overlap)::value;
    const double r = sqrt(rr), ir = 1.0 / r, irr = ir * ir;
    double t1, t2;
    pair_terms<OV>(alpha, alpha_ref, rr, r, ir, irr, t1, t2);
    if constexpr (WHOLE) {
      store_tensor(entry, b, t1, t2, sqrt(fabs(t2)) * ir, dx, dy, dz);
    } else {
      T2 t;
      t.x = (R)t1;
      t.y = (R)(t2 * irr);
      out[pair_at(k, b)] = t;
    }
  };
  auto flush = [&](int m) {
    if (lane < m) {
      const int k = queue[nq - m + lane] >> 2, b = queue[nq - m + lane] & 3;
      double dx, dy, dz;
      const double rr = image(pos[row[k]], gpos[i0 + b], dx, dy, dz);
      form(std::integral_constant<bool, true>(), whole + 16 * (size_t)k, k, b, rr, dx, dy, dz);
    }
    nq -= m;
    __syncwarp();
  };
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += 32) {
    const int k = k0 + lane, m = min(32, n - k0);
    float* entry = s_entry[WHOLE ? wl : 0] + (WHOLE ? 20 * lane : 0);
    const int j = k < n ? row[k] : 0;
    const double4 pj = pos[j];
#pragma unroll 1
    for (int b = 0; b < kGroup; b++) {
      bool near = false;
      double dx, dy, dz;
      const double4 pb = gpos[min(i0 + b, N - 1)];
      const double rr = image(pj, pb, dx, dy, dz);
      if (k < n && b < nb && j != bead_of(pb) && !(rr >= rc2)) {
        count[0] += b == 0, count[1] += b == 1, count[2] += b == 2, count[3] += b == 3;
        near = rr < 4.0;
        if (!near) form(std::integral_constant<bool, false>(), entry, k, b, rr, dx, dy, dz);
      } else if constexpr (WHOLE) {
        store_tensor(entry, b, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
      } else if (k < n) {
        T2 t;
        t.x = t.y = (R)0;
        out[pair_at(k, b)] = t;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, near);
      if (near) queue[nq + __popc(hit & ((1u << lane) - 1u))] = 4 * k + b;
      nq += __popc(hit);
    }
    __syncwarp();
    if constexpr (WHOLE) {
      float4* to = (float4*)(whole + 16 * (size_t)k0);
      for (int e = lane; e < 4 * m; e += 32)
        to[e] = ((const float4*)(s_entry[wl] + 20 * (e / 4)))[e % 4];
      __syncwarp();
    }
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
// negative where the bead's t1 carries a negative sign
__device__ __forceinline__ float2 signed_by(float2 t1, float2 a) {
  return make_float2(__uint_as_float(__float_as_uint(a.x) ^ (__float_as_uint(t1.x) << 31)),
                     __uint_as_float(__float_as_uint(a.y) ^ (__float_as_uint(t1.y) << 31)));
}

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
// set; lanes added in FP64.  Five pairs: 261 us at 50 000 beads, cutoff 14.5
// (a warp per bead, every neighbour's values read once per bead: 435), 37 us at 8000
// beads, cutoff 12.1 (50).  SPLIT warps share a group's row.
template <int NP>
struct Stage {
  static constexpr int S = 32 / NP, ITS = 32 / S, CH = S * ITS;  // entries a piece
  alignas(16) float w[16 * CH];
  int j[(CH + 3) / 4 * 4];
};

template <int NP, int SPLIT>
__global__ void __launch_bounds__(128, 4)
    k_real_apply(const int* __restrict__ cnt, const int* __restrict__ rows,
                 const float* __restrict__ rw, int cap, const float2* __restrict__ vpk, int np,
                 int p0, const double4* __restrict__ gpos, int N, int ngroup, Finish fin) {
  using V = float2;
  using P = Stage<NP>;
  constexpr int S = P::S, ITS = P::ITS, CH = P::CH, DEEP = 3, W = 25;
  constexpr int FOLD = 16 / ITS, PER = 4;  // 16-byte words an entry
  union Shared {
    P stage[4][DEEP];
    float sum[4][32 * W];
  };
  __shared__ __align__(16) unsigned char raw[sizeof(Shared)];
  Shared& sh = *reinterpret_cast<Shared*>(raw);
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * (4 / SPLIT) + wl / SPLIT, piece0 = wl % SPLIT;
  const int slot = lane / NP, pr = lane % NP;  // slot S and up: idle lanes
  __shared__ int s_bead[4][kGroup];  // the group's beads, for the results
  if (lane < kGroup) s_bead[wl][lane] = bead_of(gpos[min(kGroup * grp + lane, N - 1)]);
  V sum[2][6], part[2][6];  // beads (0, 1), (2, 3); values 3 h + c
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int e = 0; e < 6; e++) sum[b][e].x = sum[b][e].y = part[b][e].x = part[b][e].y = 0;
  if (grp < ngroup) {
    const int n = cnt[grp];
    const int* row = rows + (size_t)grp * cap;
    const float* rq = rw + 16 * (size_t)grp * cap;
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
            const float4 u = *(const float4*)(p.w + 16 * k + 8 * b),
                         v = *(const float4*)(p.w + 16 * k + 8 * b + 4);
            const V t1 = make_float2(u.x, u.y), w0 = make_float2(u.z, u.w),
                    w1 = make_float2(v.x, v.y), w2 = make_float2(v.z, v.w);
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
  float* o = sh.sum[wl] + lane * W;
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
    const int b = e / (6 * NP), p = e / 6 % NP, at = kGroup * grp + b;
    if (at >= N) break;
    const int i = s_bead[wl][b];
    double s = 0;
    for (int w = w0; w < w0 + SPLIT; w++)
      for (int u = 0; u < S; u++) s += (double)sh.sum[w][(u * NP + p) * W + 6 * b + e % 6];
    fin.write(s, p0 + p, e % 6, i);
  }
}

// ---------------------------------------------------------------------------

// The real-space sums from rows of (t1, t2 / r^2), FP64 throughout: NP packed
// pairs (p0 on), or with ONE a single right-hand side read where it lies.  One
// warp (SPLIT: that many) per group of four beads, 32 entries of the row at a
// time: the lanes form an entry's four minimum-image displacements each; for a
// single vector or pair a lane then serves its own entry, else the displacements
// go through shared memory and a lane serves one pair and every S-th entry.  The
// row streams through shared memory three pieces deep and the neighbours'
// positions (and values, NP = 1) are read a piece ahead.
template <typename R>
struct PairStage {
  alignas(16) typename Real2<R>::T t[kGroup][32];
  int j[32];
};

template <int NP, bool ONE, int SPLIT, typename R>
__global__ void __launch_bounds__(128, ONE ? 4 : 2)
    k_real_sum(Cell cell, const double4* __restrict__ pos, const double4* __restrict__ gpos,
               const int* __restrict__ cnt,
               const int* __restrict__ rows, const typename Real2<R>::T* __restrict__ rt, int cap,
               VecIn v, const double2* __restrict__ vpk, int np, int p0, int N, int ngroup,
               Finish fin) {
  using T2 = typename Real2<R>::T;
  using P = PairStage<R>;
  constexpr int S = 32 / NP, ITS = (32 + S - 1) / S, DEEP = 3, NS = ONE ? 3 : 6;
  constexpr int W = kGroup * NS + 1, WORDS = kGroup * 32 * (int)sizeof(T2) / 16;
  struct Streams {
    P stage[4][DEEP];
    double d[NP > 1 ? 4 : 1][3 * kGroup][32];  // displacements of a piece
  };
  union Shared {
    Streams in;
    double sum[4][32 * W];
  };
  __shared__ __align__(16) unsigned char raw[sizeof(Shared)];
  Shared& sh = *reinterpret_cast<Shared*>(raw);
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = blockIdx.x * (4 / SPLIT) + wl / SPLIT, piece0 = wl % SPLIT;
  const int slot = lane / NP, pr = lane % NP;  // slot S and up: idle lanes
  const int i0 = kGroup * grp;
  __shared__ int s_bead[4][kGroup];  // the group's beads, for the results
  if (lane < kGroup) s_bead[wl][lane] = bead_of(gpos[min(i0 + lane, N - 1)]);
  double sum[kGroup][NS];
#pragma unroll
  for (int b = 0; b < kGroup; b++)
#pragma unroll
    for (int e = 0; e < NS; e++) sum[b][e] = 0.0;
  if (grp < ngroup) {
    const int n = cnt[grp];
    const int* row = rows + (size_t)grp * cap;
    const T2* rq = rt + kGroup * (size_t)grp * cap;
    const size_t plane = (size_t)N * np;
    const Image image(cell);
    double4 pb[kGroup];
#pragma unroll
    for (int b = 0; b < kGroup; b++) pb[b] = gpos[min(i0 + b, N - 1)];
    P* st = sh.in.stage[wl];
    auto issue = [&](int piece, int buf) {
      const int m = min(32, n - 32 * piece);
      if (m > 0) {
        const char* from = (const char*)(rq + (size_t)kGroup * 32 * piece);
        for (int e = lane; e < WORDS; e += 32)
          copy_async((char*)st[buf].t + 16 * e, from + 16 * e, 1);
        if (lane < m) copy_async(st[buf].j + lane, row + 32 * piece + lane, 0);
      }
      copy_commit();
    };
    // a piece's gathers for this lane's entry
    struct Near {
      double4 p;
      double2 x[3];
    } cur, next;
    auto gather = [&](int piece, int buf, Near& g) {
      const int j = 32 * piece + lane < n ? st[buf].j[lane] : i0;
      g.p = pos[j];
      if constexpr (ONE) {
#pragma unroll
        for (int c = 0; c < 3; c++) g.x[c].x = v.p[c][(size_t)j * v.stride];
      } else if constexpr (NP == 1) {
#pragma unroll
        for (int c = 0; c < 3; c++) g.x[c] = __ldg(vpk + p0 + (size_t)j * np + c * plane);
      }
    };
    auto add = [&](int b, const T2& t, double dx, double dy, double dz, const double2* x) {
      const double t1 = t.x, t2 = t.y;
      double* o = sum[b];
      const double q = t2 * (dx * x[0].x + dy * x[1].x + dz * x[2].x);
      o[0] += t1 * x[0].x + q * dx;
      o[1] += t1 * x[1].x + q * dy;
      o[2] += t1 * x[2].x + q * dz;
      if constexpr (!ONE) {
        const double u = t2 * (dx * x[0].y + dy * x[1].y + dz * x[2].y);
        o[3] += t1 * x[0].y + u * dx;
        o[4] += t1 * x[1].y + u * dy;
        o[5] += t1 * x[2].y + u * dz;
      }
    };
#pragma unroll
    for (int d = 0; d < DEEP; d++) issue(piece0 + d * SPLIT, d);
    copy_wait<DEEP - 1>();
    __syncwarp();
    gather(piece0, 0, cur);
    int buf = 0;
#pragma unroll 1
    for (int piece = piece0; 32 * piece < n; piece += SPLIT) {
      copy_wait<DEEP - 2>();  // this piece and the next
      __syncwarp();
      gather(piece + SPLIT, buf + 1 == DEEP ? 0 : buf + 1, next);
      const int m = min(32, n - 32 * piece);
      const P& p = st[buf];
      if constexpr (NP == 1) {
        if (lane < m) {
#pragma unroll
          for (int b = 0; b < kGroup; b++) {
            double dx, dy, dz;
            image(cur.p, pb[b], dx, dy, dz);
            add(b, p.t[b][lane], dx, dy, dz, cur.x);
          }
        }
      } else {
        double(*d)[32] = sh.in.d[wl];
#pragma unroll
        for (int b = 0; b < kGroup; b++) {
          double dx, dy, dz;
          image(cur.p, pb[b], dx, dy, dz);
          d[3 * b][lane] = dx;
          d[3 * b + 1][lane] = dy;
          d[3 * b + 2][lane] = dz;
        }
        double2 x[ITS][3];
#pragma unroll
        for (int t = 0; t < ITS; t++) {
          const int k = t * S + slot;
          const double2* vj = vpk + p0 + pr + (size_t)(slot < S && k < m ? p.j[k] : i0) * np;
#pragma unroll
          for (int c = 0; c < 3; c++) x[t][c] = __ldg(vj + c * plane);
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < ITS; t++) {
          const int k = t * S + slot;
          if (slot < S && k < m) {
#pragma unroll
            for (int b = 0; b < kGroup; b++)
              add(b, p.t[b][k], d[3 * b][k], d[3 * b + 1][k], d[3 * b + 2][k], x[t]);
          }
        }
      }
      __syncwarp();  // the piece has been read
      issue(piece + DEEP * SPLIT, buf);
      buf = buf + 1 == DEEP ? 0 : buf + 1;
      cur = next;
    }
    copy_wait<0>();
  }
  __syncthreads();  // the streams' memory holds the sums from here on
  double* o = sh.sum[wl] + lane * W;
#pragma unroll
  for (int b = 0; b < kGroup; b++)
#pragma unroll
    for (int e = 0; e < NS; e++) o[NS * b + e] = sum[b][e];
  __syncthreads();
  if (grp >= ngroup) return;
  const int w0 = wl / SPLIT * SPLIT;
  for (int e = lane + 32 * piece0; e < NS * kGroup * NP; e += 32 * SPLIT) {
    const int b = e / (NS * NP), p = e / NS % NP;
    if (i0 + b >= N) break;
    const int i = s_bead[wl][b];
    double s = 0;
    for (int w = w0; w < w0 + SPLIT; w++)
      for (int u = 0; u < S; u++) s += sh.sum[w][(u * NP + p) * W + NS * b + e % NS];
    fin.write(s, p0 + p, e % NS, i);
  }
}

// The beads in the groups' order: cells' or, of chains, the index.
const double4* group_order(const bd_ctx* c) {
  return (const double4*)(c->rl_gpos ? c->rl_gpos : c->rl_pos);
}

// Warps a group of four beads.  More of them fill the chip sooner, fewer start fewer
// pieces.  Whole products by one, two and four, us.  FP32, whole tensors: ten
// vectors, 500 beads 69, 63, 60, 8000 207, 201, 198, 12 000 312, 301, 301, 24 000 559,
// 553, 557, 50 000 (chains of 100) 935, 935, 953; four vectors, 4000 96, 95, 95, 8000
// 128, 126, 128, 50 000 468, 472, 493; one vector, 2000 61, 59, 59, 4000 75, 75, 77, 8000
// 95, 93, 99, 16 000 142, 144, 154, 50 000 293, 302, 345.  FP64 sums: ten vectors, 8000
// 352, 337, 335, 12 000 606, 584, 584, 50 000 1825, 1829, 1875; two vectors, 2000 81, 76,
// 78, 24 000 273, 281, 304; one vector, 8000 120, 118, 120, 24 000 239, 239, 249, 50 000
// 345, 349, 376.
template <int NP, bool ONE>
int warps_of(int ng) {
  constexpr int four = 148 * (NP < 4 ? 4 : 4 * NP - 4), one = 148 * (NP == 1 && !ONE ? 24 : 40);
  return ng < four ? 4 : ng < one ? 2 : 1;
}

template <int NP, bool ONE, typename R>
void launch_sum(bd_ctx* c, int np, int p0, const Finish& fin) {
  const int ng = (c->N + kGroup - 1) / kGroup;
  const Cell cell = make_cell(c->rl_lat);
#define SUM(SPLIT_)                                                                         \
  k_real_sum<NP, ONE, SPLIT_, R><<<nblk(ng, 4 / SPLIT_), 128, 0, c->stream>>>(              \
      cell, (const double4*)c->rl_pos, group_order(c), c->rl_cnt, c->rl_rows,               \
      (const typename Real2<R>::T*)c->rl_w, c->rl_cap, fin.v, (const double2*)c->pme_vpk, np, \
      p0, c->N, ng, fin)
  switch (warps_of<NP, ONE>(ng)) {
    case 4: SUM(4); break;
    case 2: SUM(2); break;
    default: SUM(1);
  }
#undef SUM
}

template <int NP>
void launch_apply(bd_ctx* c, int np, int p0, const Finish& fin) {
  const int ng = (c->N + kGroup - 1) / kGroup;
#define REAL(SPLIT_)                                                                      \
  k_real_apply<NP, SPLIT_><<<nblk(ng, 4 / SPLIT_), 128, 0, c->stream>>>(                  \
      c->rl_cnt, c->rl_rows, (const float*)c->rl_w, c->rl_cap, (const float2*)c->pme_vpk, \
      np, p0, group_order(c), c->N, ng, fin)
  switch (warps_of<NP, false>(ng)) {
    case 4: REAL(4); break;
    case 2: REAL(2); break;
    default: REAL(1);
  }
#undef REAL
}

// In passes of up to five pairs.
template <class F>
void by_fives(bd_ctx* c, int np, F launch) {
  for (int p0 = 0; p0 < np; p0 += 5) {
    c->launches++;
    switch (std::min(5, np - p0)) {
      case 1: launch(std::integral_constant<int, 1>(), p0); break;
      case 2: launch(std::integral_constant<int, 2>(), p0); break;
      case 3: launch(std::integral_constant<int, 3>(), p0); break;
      case 4: launch(std::integral_constant<int, 4>(), p0); break;
      default: launch(std::integral_constant<int, 5>(), p0);
    }
  }
}

// Rows hold whole tensors (FP32 contexts with noise blocks) or (t1, t2 / r^2).
bool whole_tensors(const bd_ctx* c) { return c->pme_f32 && c->nbk > 1; }

}  // namespace

namespace bd {

constexpr int kRowCells = 4096;  // most cells of the rows' search

// Rows of cap entries for every group; without memory for them there are none
// (rl_rows null) and the mobility is not built.
static int rows_alloc(bd_ctx* c, int cap) {
  size_t ng = ((size_t)c->N + kGroup - 1) / kGroup, old = (size_t)c->rl_cap;
  size_t tensor = whole_tensors(c) ? 16 : c->pme_f32 ? 8 : 16, each = 4 + tensor * kGroup;
  cap = (cap + 31) / 32 * 32;
  if (c->rl_rows) {
    CU(cudaStreamSynchronize(c->stream));
    free_all({&c->rl_rows, &c->rl_w});
    c->bytes -= each * ng * old;
  }
  c->rl_cap = 0;
  int s = alloc_all(c, {{&c->rl_rows, 4 * ng * cap}, {&c->rl_w, tensor * kGroup * ng * cap}});
  if (s == BD_OK) c->rl_cap = cap;
  return s;
}

// Entries of a row before any have overflowed: an explicit cap per bead, or 2.5
// times the mean number of beads within the cutoff at the system's density, at
// least 512.  Rows that overflow it are grown; no row is longer than N, nor with
// an explicit cap than four beads' pairs.
static int first_cap(const bd_ctx* c) {
  const double mean = 4.0 / 3.0 * M_PI * c->pme_rc * c->pme_rc * c->pme_rc * c->N / c->boxvol;
  const int cap = c->p.pme_max_pairs > 0 ? c->p.pme_max_pairs : std::max(512, (int)ceil(2.5 * mean));
  return std::min(cap, std::max(c->N, 1));
}

// The rows of a first preparation, or of one after rows that could not be grown.
int real_rows(bd_ctx* c) { return c->rl_rows ? BD_OK : rows_alloc(c, first_cap(c)); }

int real_alloc(bd_ctx* c) {
  const size_t N = c->N;
  // as many cells as the groups' order has where beads are not chained
  const bool order = !by_index(c->Nb);
  c->rl_ncell_cap = order ? (int)std::max((size_t)kRowCells, 2 * N) : kRowCells;
  int s;
  if (order && (s = alloc_all(c, {{&c->rl_gpos, 32 * N}})) != BD_OK) return s;
  s = alloc_all(c, {{&c->rl_cnt, 4 * N},
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
  free_all({&c->rl_rows, &c->rl_w, &c->rl_gpos, &c->rl_cnt, &c->rl_need, &c->rl_cell_of, &c->rl_spos,
            &c->rl_beads, &c->rl_cell_count, &c->rl_cell_start, &c->rl_cursor});
  c->rl_cap = 0;
}

// The beads by cells of geometry g (reduced to at most `most` cells) in rl_beads,
// the cells' ranges in rl_cell_start; returns their number.
static int bin_beads(bd_ctx* c, const Cell& cell, RGeom& g, int most, double cr, double sr) {
  const int N = c->N;
  while ((long)g.n[0] * g.n[1] * g.n[2] > most) {
    int d = g.n[0] >= g.n[1] && g.n[0] >= g.n[2] ? 0 : (g.n[1] >= g.n[2] ? 1 : 2);
    g.n[d]--;
  }
  const int ncell = g.n[0] * g.n[1] * g.n[2];
  c->launches += 3;
  k_rl_count<<<nblk(N, 256), 256, 0, c->stream>>>(cell, g, c->rx, c->ry, c->rz, cr, sr, N,
                                                  c->rl_cell_of, c->rl_cell_count);
  k_rl_scan<<<1, 1024, 0, c->stream>>>(ncell, c->rl_cell_count, c->rl_cell_start, c->rl_cursor);
  k_rl_fill<<<nblk(N, 256), 256, 0, c->stream>>>(c->rl_cell_of, c->rl_cell_start, c->rl_cursor,
                                                 c->rl_beads, N);
  return ncell;
}

// The groups' rows for the positions in rl_pos (lab frame; rx, ry, rz and the
// rotation (cr, sr) give the same); alpha_ref is calcHI's split parameter.
int real_prepare(bd_ctx* c, const Lat& l, const Cell& cell, double cr, double sr,
                 double alpha_ref) {
  int s, N = c->N;
  double rc = c->pme_rc, alpha = c->pme_alpha;
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
  if (c->rl_gpos) {
    // the groups' order: columns of four beads' mean width, cut so that a cell
    // holds one bead
    const double h = cbrt(4.0 * cell.V / N);
    RGeom o;
    for (int d = 0; d < 3; d++) o.n[d] = std::max(1, (int)(w[d] / (d < 2 ? h : 0.25 * h)));
    const int n = bin_beads(c, cell, o, c->rl_ncell_cap, cr, sr);
    c->launches++;
    k_rl_group<<<nblk(n, 8), 256, 0, c->stream>>>(c->rl_cell_start, n, c->rl_beads,
                                                  (const double4*)c->rl_pos, (double4*)c->rl_gpos);
  }
  const int ncell = bin_beads(c, cell, g, kRowCells, cr, sr);
  c->launches++;
  k_rl_order<<<ncell, 256, 0, c->stream>>>(c->rl_cell_start, c->rl_beads,
                                           (const double4*)c->rl_pos, (double4*)c->rl_spos);
  if ((s = launch_ok(c)) != BD_OK) return s;
  // the rows; those that overflow are grown to 1.25 times the longest one and
  // built again, an error where they must not be longer
  const int ng = (N + kGroup - 1) / kGroup;
  const int most = c->p.pme_max_pairs > 0
                       ? (int)std::min((long)N, (long)kGroup * c->p.pme_max_pairs)
                       : N;
  for (bool grow = c->rl_cap < most;; grow = false) {
    c->launches++;
    k_rl_find<<<nblk(ng, 4), 128, 0, c->stream>>>(
        cell, g, group_order(c), N, ng, c->rl_cell_start, (const double4*)c->rl_spos,
        rc * rc, c->rl_cap, c->rl_cnt, c->rl_rows, grow ? c->rl_need : nullptr, c->err);
    if (!grow) break;
    int longest = 0;
    CU(cudaMemcpyAsync(&longest, c->rl_need, 4, cudaMemcpyDeviceToHost, c->stream));
    if ((s = check(c)) != BD_OK) return s;
    if (longest <= c->rl_cap) break;
    CU(cudaMemsetAsync(c->rl_need, 0, 4, c->stream));
    if ((s = rows_alloc(c, std::min(most, (int)ceil(1.25 * longest)))) != BD_OK) return s;
  }
  c->launches++;
#define TENSORS(...)                                                                          \
  k_rl_tensors<__VA_ARGS__><<<nblk(ng, 4), 128, 0, c->stream>>>(                              \
      cell, (const double4*)c->rl_pos, group_order(c), N, ng, c->rl_cnt, c->rl_rows, c->rl_cap, \
      rc * rc, alpha, alpha_ref, c->p.pme_max_pairs, c->rl_w, c->err)
  if (whole_tensors(c))
    TENSORS(float, true);
  else if (c->pme_f32)
    TENSORS(float, false);
  else
    TENSORS(double, false);
#undef TENSORS
  c->rl_lat = l;
  return launch_ok(c);
}

int real_apply(bd_ctx* c, int np, const Finish& fin) {
  if (whole_tensors(c)) {
    by_fives(c, np, [&](auto n, int p0) { launch_apply<decltype(n)::value>(c, np, p0, fin); });
  } else if (fin.k == 1) {
    c->launches++;
    if (c->pme_f32)
      launch_sum<1, true, float>(c, np, 0, fin);
    else
      launch_sum<1, true, double>(c, np, 0, fin);
  } else {  // FP64: FP32 contexts without noise blocks have one right-hand side
    by_fives(c, np, [&](auto n, int p0) {
      launch_sum<decltype(n)::value, false, double>(c, np, p0, fin);
    });
  }
  return launch_ok(c);
}

}  // namespace bd
