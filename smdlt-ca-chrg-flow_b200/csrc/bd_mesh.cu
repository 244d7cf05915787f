// Spreading and interpolation of the particle-mesh mobility without atomics.
//
// No counterpart in the reference (see bd_pme.cu).  Grids hold, per packed
// pair of right-hand sides, K^3 points of three complex components, the
// component fastest; where cuFFT transforms them (pme_planar), the components one
// after the other, and a single right-hand side's grid is real.
//
// Spreading: the grid is cut into columns of CY x CZ points in (y, z), running
// along x.  A warp owns a column (or a segment of it) for NG packed pairs, a
// lane per (y, z) and pair: it walks the beads whose stencil meets the column
// in order of their base index along x, holding the P grid levels that the
// current base reaches in registers.  A bead's P x-weights times the lane's y
// and z weights and the bead's values are added to those levels; a level is
// written when the walk has passed it (every point is written exactly once, so
// the grid needs no clearing), and the window shifts.
// An order-8 stencil covers 8 x 8 of the (y, z) plane and meets (7 + CY)(7 +
// CZ)/(CY CZ) columns, so small columns waste fewer lanes (the share of them
// inside the stencil is 39 % at 4 x 8, 71 % at 2 x 3) as long as the warp's
// other lanes serve other pairs: 5 pairs by 2 x 3, 4 by 2 x 4, 3 by 2 x 5, 2 by
// 4 x 4, 1 by 4 x 8.
// Bound by the FP32 (FP64) pipe and the issue of its instructions: 48 (P = 8)
// multiply-adds per lane and bead, two at a time (fma.rn.f32x2) in FP32, next
// to about 20 others.
// Five pairs, order 8: 153 us at 50 000 beads on 100^3 (one complex L2 atomic
// per stencil point, component and pair took about 400), 41 us at 8000 beads on
// 64^3 (74); FP64 66 us there (385).
//
// Interpolation: a warp per bead and pair reads the stencil's 64 rows of 24
// complex values (192 contiguous bytes, FP32), a lane the same third of a row
// position throughout, so its y and z weights and addresses stay in registers.
// Bound by L1 throughput.
// Five pairs, order 8: 245 us at 50 000 beads on 100^3 (separate component
// grids, 64 bytes a row: about 300), 39 us at 8000 beads on 64^3 (54); FP64 70 us
// there.
//
// The columns' lists are built once per mobility build (the positions are
// frozen until the next): per column and base index the beads in increasing
// index, so the sums are formed in a fixed order and a product is
// reproducible bit by bit.
#include <algorithm>
#include <type_traits>

#include "bd_ctx.cuh"
#include "bd_cell.cuh"
#include "bd_mesh.cuh"

using namespace bd;

#define CU(call) BD_CU(call)

namespace {

constexpr int kMaxTouched = 8;  // columns that a stencil can meet along y or z

// The distinct column indices of size-w cells that the rows b, b - 1, ..,
// b - P + 1 (modulo K) lie in.
__device__ __forceinline__ int touched(int b, int P, int K, int w, int* out) {
  int n = 0, last = -1;
  for (int d = 0; d < P; d++) {
    int y = b - d;
    y += y < 0 ? K : 0;
    int c = y / w;
    if (c == last) continue;
    last = c;
    bool seen = false;
    for (int q = 0; q < n; q++) seen |= out[q] == c;
    if (!seen) out[n++] = c;
  }
  return n;
}

// Beads per (column, base index); with ent also their entries from bin[] on.
__global__ void k_mesh_list(const int* __restrict__ base, int N, int K, int P, int CY, int CZ,
                            int npz, int* count, const int* __restrict__ bin, int* ent) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int cy[kMaxTouched], cz[kMaxTouched];
  int ny = touched(base[3 * i + 1], P, K, CY, cy);
  int nz = touched(base[3 * i + 2], P, K, CZ, cz);
  for (int a = 0; a < ny; a++)
    for (int b = 0; b < nz; b++) {
      size_t q = (size_t)(cy[a] * npz + cz[b]) * K + base[3 * i];
      int at = atomicAdd(count + q, 1);
      if (ent) ent[bin[q] + at] = i;
    }
}

// Each bin in increasing bead index (bins hold a few beads).
__global__ void k_mesh_sort(const int* __restrict__ bin, size_t nbin, int* ent) {
  size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbin) return;
  int lo = bin[b], hi = bin[b + 1];
  for (int a = lo + 1; a < hi; a++) {
    int v = ent[a], q = a - 1;
    for (; q >= lo && ent[q] > v; q--) ent[q + 1] = ent[q];
    ent[q + 1] = v;
  }
}

// Exclusive scan of a[0 .. n) in place, the total at a[n]: 2048 entries per
// block, the block totals scanned by one block in between.
constexpr int kScanBlock = 2048;

__device__ __forceinline__ int block_scan_excl(int v, int* sh, int& total) {
  int t = threadIdx.x, lane = t & 31, w = t >> 5, in = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int x = __shfl_up_sync(0xffffffffu, in, o);
    if (lane >= o) in += x;
  }
  if (lane == 31) sh[w] = in;
  __syncthreads();
  int before = 0;
  total = 0;
  for (int q = 0; q < (int)(blockDim.x >> 5); q++) {
    if (q < w) before += sh[q];
    total += sh[q];
  }
  __syncthreads();
  return before + in - v;
}

__global__ void __launch_bounds__(256) k_scan_sums(const int* __restrict__ a, size_t n, int* sums) {
  __shared__ int sh[8];
  size_t lo = (size_t)blockIdx.x * kScanBlock;
  int s = 0, total;
  for (int q = threadIdx.x; q < kScanBlock; q += 256)
    if (lo + q < n) s += a[lo + q];
  block_scan_excl(s, sh, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_blocks(int* sums, int nb, int* total_out) {
  __shared__ int sh[32];
  int run = 0;
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    int b = b0 + threadIdx.x, v = b < nb ? sums[b] : 0, total;
    int e = block_scan_excl(v, sh, total);
    if (b < nb) sums[b] = run + e;
    run += total;
  }
  if (threadIdx.x == 0) *total_out = run;
}

__global__ void __launch_bounds__(256) k_scan_place(int* a, size_t n, const int* __restrict__ sums) {
  __shared__ int sh[8];
  size_t lo = (size_t)blockIdx.x * kScanBlock + threadIdx.x * 8;
  int v[8], s = 0, total;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    v[q] = lo + q < n ? a[lo + q] : 0;
    s += v[q];
  }
  int run = sums[blockIdx.x] + block_scan_excl(s, sh, total);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    if (lo + q < n) a[lo + q] = run;
    run += v[q];
  }
}

// The values of the packed pairs for the spreading and the real-space sums:
// component c of pair p (both right-hand sides) at vpk[(c N + i) np + p], a
// bead's pairs side by side.
template <typename T>
__global__ void k_mesh_pack(VecIn v, size_t vr, int k, int np, int N, T* vpk) {
  using R = decltype(vpk->x);
  const int i = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
  if (i >= N) return;
  const size_t oa = (size_t)(2 * p) * vr + (size_t)i * v.stride;
  const bool two = 2 * p + 1 < k;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    T x;
    x.x = (R)v.p[c][oa];
    x.y = two ? (R)v.p[c][oa + vr] : (R)0;
    vpk[((size_t)c * N + i) * np + p] = x;
  }
}

// ---------------------------------------------------------------------------

template <typename R>
struct GridVal;
template <>
struct GridVal<float> {
  using T = float2;
  using W = float2;  // a weight in both halves, as fma.rn.f32x2 wants it
};
template <>
struct GridVal<double> {
  using T = double2;
  using W = double;
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d, x = *reinterpret_cast<unsigned long long*>(&a),
                        y = *reinterpret_cast<unsigned long long*>(&b),
                        z = *reinterpret_cast<unsigned long long*>(&c);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ void madd(float2 w, float2 x, float2& a) { a = fma2(w, x, a); }
__device__ __forceinline__ void madd(double w, double2 x, double2& a) {
  a.x = fma(w, x.x, a.x);
  a.y = fma(w, x.y, a.y);
}
__device__ __forceinline__ void madd(float w, float x, float& a) { a = fmaf(w, x, a); }
__device__ __forceinline__ void madd(double w, double x, double& a) { a = fma(w, x, a); }
// grid values into FP64 sums
__device__ __forceinline__ void madd(double w, float2 x, double2& a) {
  a.x = fma(w, (double)x.x, a.x);
  a.y = fma(w, (double)x.y, a.y);
}
__device__ __forceinline__ void madd(double w, float x, double& a) { a = fma(w, (double)x, a); }
// a weight as the sums of V take it
template <typename V, typename R>
__device__ __forceinline__ auto weight(R x) {
  if constexpr (std::is_same_v<V, float2>)
    return make_float2(x, x);
  else
    return x;
}
__device__ __forceinline__ void put(float2& w, float x) { w = make_float2(x, x); }
__device__ __forceinline__ void put(float& w, float x) { w = x; }
__device__ __forceinline__ void put(double& w, double x) { w = x; }
// Accumulated values: a complex pair, or a real number where a single
// right-hand side leaves the imaginary parts zero.
__device__ __forceinline__ void zero(float& a) { a = 0.f; }
__device__ __forceinline__ void zero(double& a) { a = 0.0; }
__device__ __forceinline__ void zero(float2& a) { a = make_float2(0.f, 0.f); }
__device__ __forceinline__ void zero(double2& a) { a = make_double2(0.0, 0.0); }
__device__ __forceinline__ float2 as_pair(float a) { return make_float2(a, 0.f); }
__device__ __forceinline__ double2 as_pair(double a) { return make_double2(a, 0.0); }
__device__ __forceinline__ float2 as_pair(float2 a) { return a; }
__device__ __forceinline__ double2 as_pair(double2 a) { return a; }
__device__ __forceinline__ float scaled(float w, float a) { return w * a; }
__device__ __forceinline__ double scaled(double w, double a) { return w * a; }
__device__ __forceinline__ float2 scaled(float w, float2 a) { return make_float2(w * a.x, w * a.y); }
__device__ __forceinline__ double2 scaled(double w, double2 a) {
  return make_double2(w * a.x, w * a.y);
}
__device__ __forceinline__ void set_pair(float2& f, float x, float y) { f = make_float2(x, y); }
__device__ __forceinline__ void set_pair(double2& f, double x, double y) { f = make_double2(x, y); }
__device__ __forceinline__ void set_pair(float& f, float x, float) { f = x; }
__device__ __forceinline__ void set_pair(double& f, double x, double) { f = x; }

// One bead of a column's walk in shared memory: x-weights from the lowest
// level up, the (y, z) weights of the column's points (products of FP64 weights,
// rounded once), the pairs' values, the base index along x.  Padded to an odd number of 16-byte words, so that
// the lanes of a warp store their records without bank conflicts.
template <int P, typename R, int NG, int CY, int CZ, bool ONE>
struct RecData {
  std::conditional_t<ONE, R, typename GridVal<R>::W> wx[P];
  std::conditional_t<ONE, R, typename GridVal<R>::T> f[NG][3];
  double wy[NG == 1 ? CY : 1], wz[NG == 1 ? CZ : 1];
  R wyz[NG == 1 ? 1 : CY * CZ];
  int at;
};
template <typename S>
struct alignas(16) Rec : S {
  static constexpr int words = (int)((sizeof(S) + 15) / 16);
  char fill[16 * (words + (words % 2 == 0 ? 1 : 0)) - sizeof(S)];
};

// The weights along x in the grid's type: FP32 ones are kept beside the FP64 ones
// (converted by every warp that meets the bead, spreading and interpolation of the five
// pairs above took 163 and 253 us).
__device__ __forceinline__ const float* level_weights(const float* wx, const double*, int i) {
  return wx + (size_t)i * kMaxOrder;
}
__device__ __forceinline__ const double* level_weights(const double*, const double* w, int i) {
  return w + (size_t)i * 3 * kMaxOrder;
}

struct SpreadArgs {
  const int* base;
  const double* w;  // 8 weights per bead and direction
  const void* wx;   // the first direction's in the grid's type
  const int* ent;
  const int* bin;
  int K, npz, npatch, nseg, nset, np, N;
  const void* vpk;  // packed values
  int ps;           // grid layout: a point's, a component's stride
  size_t cs;
};

template <int P, typename R, int NG, int CY, int CZ, bool ONE>
__global__ void __launch_bounds__(32, sizeof(R) == 4 ? 16 : 8)
    k_mesh_spread(SpreadArgs m, R* grid) {
  using T = typename GridVal<R>::T;
  using V = std::conditional_t<ONE, R, T>;
  using S = Rec<RecData<P, R, NG, CY, CZ, ONE>>;
  static_assert(NG * CY * CZ <= 32, "a lane per point and pair");
  // a warp per block: columns differ in their beads by a factor of two and
  // more, and single warps leave the fewest idle slots behind
  __shared__ S s_rec[32];
  const int lane = threadIdx.x, job = blockIdx.x;
  // columns fastest: the neighbours along z of a block complete its sectors
  const int patch = job % m.npatch, seg = job / m.npatch % m.nseg,
            set = job / (m.npatch * m.nseg);
  const int K = m.K, xs = (int)((long long)seg * K / m.nseg),
            xe = (int)((long long)(seg + 1) * K / m.nseg);
  const int y0 = patch / m.npz * CY, z0 = patch % m.npz * CZ;
  const int g = lane / (CY * CZ) < NG ? lane / (CY * CZ) : 0;
  const int ly = lane % (CY * CZ) / CZ, lz = lane % CZ;
  const int pr = set * NG + g;
  const bool own = lane < NG * CY * CZ && pr < m.np && y0 + ly < K && z0 + lz < K;
  const size_t K2 = (size_t)K * K;
  const size_t here = (size_t)(y0 + ly) * K + (z0 + lz);
  T* out = (T*)grid + 3 * (size_t)(own ? pr : 0) * K2 * K + here * m.ps;
  // bases xs .. xe + P - 2, wrapped: entries [e0, e0 + n0), then [f0, f0 + n1)
  const int* bin = m.bin + (size_t)patch * K;
  const int top = xe + P - 1;
  const int e0 = bin[xs], n0 = bin[min(K, top)] - e0;
  const int f0 = bin[0], n1 = top > K ? bin[top - K] - f0 : 0;
  const int n = n0 + n1;
  V acc[P][3];
#pragma unroll
  for (int a = 0; a < P; a++)
#pragma unroll
    for (int c = 0; c < 3; c++) zero(acc[a][c]);
  int lo = xs - (P - 1);  // grid level of acc[0]
  auto advance = [&]() {
    if (lo >= xs && own) {
      if (ONE && m.ps == 1) {
        R* o = grid + here + K2 * (size_t)lo;
#pragma unroll
        for (int c = 0; c < 3; c++) o[c * m.cs] = as_pair(acc[0][c]).x;
      } else {
        T* o = out + m.ps * K2 * (size_t)lo;
#pragma unroll
        for (int c = 0; c < 3; c++) o[c * m.cs] = as_pair(acc[0][c]);
      }
    }
#pragma unroll
    for (int a = 0; a + 1 < P; a++)
#pragma unroll
      for (int c = 0; c < 3; c++) acc[a][c] = acc[a + 1][c];
#pragma unroll
    for (int c = 0; c < 3; c++) zero(acc[P - 1][c]);
    lo++;
  };
  // records straight into shared memory; only the next batch's bead indices are
  // read ahead (the other warps of the SM cover the records' latency, and the
  // registers go to the window)
  auto entry = [&](int t) { return t >= n ? 0 : t < n0 ? m.ent[e0 + t] : m.ent[f0 + t - n0]; };
  auto stage = [&](int t, int i) {
    if (t >= n) return;
    S& r = s_rec[lane];
    const double* w = m.w + (size_t)i * 3 * kMaxOrder;
    const R* wx = level_weights((const R*)m.wx, m.w, i);
    const int b1 = m.base[3 * i + 1], b2 = m.base[3 * i + 2];
    r.at = m.base[3 * i] + (t < n0 ? 0 : K);
#pragma unroll
    for (int a = 0; a < P; a++) put(r.wx[a], wx[P - 1 - a]);
    double wz[CZ];
#pragma unroll
    for (int q = 0; q < CZ; q++) {
      int d = b2 - (z0 + q);
      d += d < 0 ? K : 0;
      wz[q] = d < P && z0 + q < K ? w[2 * kMaxOrder + d] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < CY; q++) {
      int d = b1 - (y0 + q);
      d += d < 0 ? K : 0;
      const double wy = d < P && y0 + q < K ? w[kMaxOrder + d] : 0.0;
      if constexpr (NG == 1) {
        r.wy[q] = wy;
      } else {
#pragma unroll
        for (int e = 0; e < CZ; e++) r.wyz[q * CZ + e] = (R)(wy * wz[e]);
      }
    }
    if constexpr (NG == 1) {
#pragma unroll
      for (int e = 0; e < CZ; e++) r.wz[e] = wz[e];
    }
#pragma unroll
    for (int u = 0; u < NG; u++) {
      const int p = min(set * NG + u, m.np - 1);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const T a = ((const T*)m.vpk)[((size_t)c * m.N + i) * m.np + p];
        set_pair(r.f[u][c], a.x, a.y);
      }
    }
  };
  int bead = entry(lane);
  for (int t0 = 0; t0 < n; t0 += 32) {
    __syncwarp();
    stage(t0 + lane, bead);
    bead = entry(t0 + 32 + lane);
    __syncwarp();
    const int nb = min(32, n - t0);
#pragma unroll 1
    for (int u = 0; u < nb; u++) {
      const S& q = s_rec[u];
      R wyz;
      if constexpr (NG == 1)
        wyz = (R)(q.wy[ly] * q.wz[lz]);
      else
        wyz = q.wyz[ly * CZ + lz];
      V t[3];
#pragma unroll
      for (int c = 0; c < 3; c++) t[c] = scaled(wyz, q.f[g][c]);
      const int want = q.at - (P - 1);
#pragma unroll 1
      while (lo < want) advance();
#pragma unroll
      for (int a = 0; a < P; a++) {
        const auto wx = q.wx[a];
#pragma unroll
        for (int c = 0; c < 3; c++) madd(wx, t[c], acc[a][c]);
      }
    }
  }
#pragma unroll 1
  while (lo < xe) advance();
}

// val[(pr N + i) 6 + 3 h + c] = sum_g W_i(g) grid (h: real, imaginary part):
// a warp per bead and pair.  The stencil's 3 P^3 complex values are taken 32 at
// a time in memory order (rows of P points along z, three components each);
// 96 values are a whole number of points, so load t of a lane always holds
// component (2 t + lane) mod 3: one sum for each t mod 3, put in component
// order at the end.  Order 8 takes a lane's sums along x (8 levels) in the grid's
// type and the rest in FP64: 245 us for the five pairs above, 404 with every FP32
// value converted (four a clock and quarter of an SM), 448 with FP32 sums that keep
// what they round away.  The product's error against FP64, geometric mean of 12
// systems of 900 to 32 000 beads, ten vectors: 1.34e-7, 1.33e-7 by those last two
// (1.89e-7 by atomics, cuFFT and FP64 sums of every term, 1.40e-7 with FP32 weights
// and lanes).
// A single right-hand side's values are real: they fill planar real grids (kReal) or
// are the real parts of an interleaved one (kSingle; with the zero imaginary parts an
// iteration of a 4000-bead solve on 64^3 FP64 took 120.7 us, 114.0 without).
enum Layout { kInterleaved, kSingle, kPlanar, kReal };

template <int P, typename R, Layout LAY>
__global__ void __launch_bounds__(256)
    k_mesh_gather(const int* __restrict__ base, const double* __restrict__ w,
                  const R* __restrict__ wxs,
                  const R* __restrict__ grid, int N, int K, double* __restrict__ val) {
  using T = typename GridVal<R>::T;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, pr = blockIdx.y;
  if (i >= N) return;
  const double* w0 = w + (size_t)i * 3 * kMaxOrder;
  const double* w1 = w0 + kMaxOrder;
  const double* w2 = w1 + kMaxOrder;
  // a single vector's warp converts its own: 49 us for 50 000 beads, 54 with the loads
  const R* wl = level_weights(wxs, w, i);
  const int b0 = base[3 * i], b1 = base[3 * i + 1], b2 = base[3 * i + 2];
  const size_t K2 = (size_t)K * K;
  constexpr bool RE = LAY == kSingle || LAY == kReal, INTER = LAY == kInterleaved || LAY == kSingle;
  constexpr int ps = INTER ? 3 : 1, es = LAY == kSingle ? 2 : 1;
  const size_t cs = INTER ? 1 : K2 * K;
  using V = std::conditional_t<RE, R, T>;
  using S = std::conditional_t<RE, double, double2>;
  const V* gp = (const V*)grid + (size_t)pr * 3 * K2 * K;  // pair 0 where RE
  S s[3];
#pragma unroll
  for (int j = 0; j < 3; j++) zero(s[j]);
  constexpr bool own_sums = P == 8 && !INTER;  // component c in sum c
  if constexpr (own_sums) {
    // four rows of one component a load
    unsigned off[2];
    double wyz[2];
    V u[2][3];
    int gz = b2 - (P - 1) + lane % 8;
    gz += gz < 0 ? K : 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      int gy = b1 - (4 * h + lane / 8);
      gy += gy < 0 ? K : 0;
      off[h] = (unsigned)(gy * K + gz);
      wyz[h] = w1[4 * h + lane / 8] * w2[P - 1 - lane % 8];
#pragma unroll
      for (int j = 0; j < 3; j++) zero(u[h][j]);
    }
#pragma unroll
    for (int a = 0; a < P; a++) {
      int gx = b0 - a;
      gx += gx < 0 ? K : 0;
      const V* gl = gp + K2 * (size_t)gx;
      const auto wx = weight<V>(RE ? (R)w0[a] : wl[a]);
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 3; j++) madd(wx, gl[off[h] + (size_t)j * cs], u[h][j]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int j = 0; j < 3; j++) madd(wyz[h], u[h][j], s[j]);
  } else if constexpr (P == 8) {
    // four rows in three loads; rows 4 q + (0..3) of x level q / 2: the lane's
    // point and its offset within (y, z) depend on q only by its parity
    int off[3][2];
    double wyz[3][2];
    V u[3][2];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int f = 32 * j + lane, ro = f / 24, z = f % 24 / 3;
      int gz = b2 - (P - 1) + z;
      gz += gz < 0 ? K : 0;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int gy = b1 - (4 * h + ro);
        gy += gy < 0 ? K : 0;
        off[j][h] = (gy * K + gz) * 3 + f % 3;
        wyz[j][h] = w1[4 * h + ro] * w2[P - 1 - z];
        zero(u[j][h]);
      }
    }
#pragma unroll
    for (int a = 0; a < P; a++) {
      int gx = b0 - a;
      gx += gx < 0 ? K : 0;
      const V* gl = gp + es * 3 * K2 * (size_t)gx;
      const auto wx = weight<V>(RE ? (R)w0[a] : wl[a]);
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
          if constexpr (sizeof(R) == 4)
            madd(wx, gl[es * off[j][h]], u[j][h]);
          else  // fewer sums to hold: 4000 beads 10.6 us a pair, not 14.2
            madd(wx * wyz[j][h], gl[es * off[j][h]], s[j]);
        }
    }
    if constexpr (sizeof(R) == 4) {
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 3; j++) madd(wyz[j][h], u[j][h], s[j]);
    }
  } else {
#pragma unroll 1
    for (int t0 = 0; 32 * t0 < 3 * P * P * P; t0 += 3) {
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const int f = 32 * (t0 + j) + lane;
        if (f >= 3 * P * P * P) break;
        const int z = f / 3 % P, row = f / (3 * P), b = row % P, a = row / P;
        int gx = b0 - a, gy = b1 - b, gz = b2 - (P - 1) + z;
        gx += gx < 0 ? K : 0;
        gy += gy < 0 ? K : 0;
        gz += gz < 0 ? K : 0;
        madd(w0[a] * w1[b] * w2[P - 1 - z],
             gp[es * (ps * ((size_t)gx * K2 + (size_t)gy * K + gz) + (f % 3) * cs)], s[j]);
      }
    }
  }
  // component c is in sum 2 (c - lane) mod 3
  const int r = own_sums ? -1 : lane % 3;
  const S c0 = r <= 0 ? s[0] : r == 1 ? s[1] : s[2];
  const S c1 = r < 0 ? s[1] : r == 0 ? s[2] : r == 1 ? s[0] : s[1];
  const S c2 = r < 0 ? s[2] : r == 0 ? s[1] : r == 1 ? s[2] : s[0];
  if constexpr (RE) {
    double x[3] = {c0, c1, c2};
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
    if (lane < 3) val[(size_t)i * 6 + lane] = lane == 0 ? x[0] : lane == 1 ? x[1] : x[2];
  } else {
    // real parts to the lower, imaginary parts to the upper half of the warp
    const bool up = lane & 16;
    double x[3] = {up ? c0.y : c0.x, up ? c1.y : c1.x, up ? c2.y : c2.x};
    const double y[3] = {up ? c0.x : c0.y, up ? c1.x : c1.y, up ? c2.x : c2.y};
#pragma unroll
    for (int c = 0; c < 3; c++) {
      x[c] += __shfl_xor_sync(0xffffffffu, y[c], 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
    }
    const int e = lane & 15;
    if (e < 3) val[((size_t)pr * N + i) * 6 + (up ? 3 : 0) + e] = e == 0 ? x[0] : e == 1 ? x[1] : x[2];
  }
}

// ---------------------------------------------------------------------------

// Columns of the layouts, by the number of pairs a warp serves.
constexpr int kCols[6][2] = {{0, 0}, {4, 8}, {4, 4}, {2, 5}, {2, 4}, {2, 3}};

// Work of a spreading of np pairs in layout ng: bead visits times warps.
double layout_cost(int np, int ng, int P) {
  double cy = kCols[ng][0], cz = kCols[ng][1];
  return (P - 1 + cy) * (P - 1 + cz) / (cy * cz) * ((np + ng - 1) / ng);
}

// Few beads for the grid's points: writing the points is most of the work, and the
// layout of one pair a warp writes the longest runs.  Ten vectors by it and by five
// pairs a warp, us, FP32: 144^3 1000 beads 965 and 1080, 32 000 1217 and 1333, 50 000
// 1425 and 1464; 100^3 8000 beads 408 and 420, 16 000 502 and 485, 50 000 1010 and 937.
// FP64: 144^3 8000 beads 1720 and 1873, 32 000 2252 and 2276, 50 000 2705 and 2618;
// 100^3 8000 beads 752 and 742.
// On 64^3 and below, 500 FP32 beads on 32^3 for one, five pairs a warp are faster at
// any density (10.7 us and 14.7).
bool sparse(const bd_ctx* c) {
  const size_t K = c->pmeK;
  return K >= 90 && (size_t)c->N * (c->pme_f32 ? 64 : 128) < K * K * K;
}

// Segments of a column: about 14 warps on every SM (16 fit), none shorter than
// half a stencil (a segment repeats P - 1 levels of its beads).  Segments
// measured, us: 1700 columns of 100 levels 1: 154, 2: 159, 3: 155, 6: 163; 704
// columns of 64 levels 1: 56, 2: 45, 3: 42, 4: 43, 6: 46.
int segments(int K, int njob) {
  int want = (148 * 14 + njob / 2) / njob;
  return std::max(1, std::min(want, K / 4));
}

size_t patches(int K, int ng) {
  return (size_t)((K + kCols[ng][0] - 1) / kCols[ng][0]) *
         ((K + kCols[ng][1] - 1) / kCols[ng][1]);
}

// Columns that a stencil can meet: P rows over cells of w, one more where the
// last cell is short.
int most_touched(int K, int P, int w) {
  return std::min((P + w - 2) / w + 1 + (K % w ? 1 : 0), (K + w - 1) / w);
}

template <int P, typename R>
void launch_spread(bd_ctx* c, int k, int ng, int nb, const SpreadArgs& m, R* grid) {
#define SPREAD(...) \
  k_mesh_spread<P, R, __VA_ARGS__><<<nb, 32, 0, c->stream>>>(m, grid)
  switch (ng) {
    case 1:
      if (k == 1)
        SPREAD(1, 4, 8, true);
      else
        SPREAD(1, 4, 8, false);
      break;
    case 2: SPREAD(2, 4, 4, false); break;
    case 3: SPREAD(3, 2, 5, false); break;
    case 4: SPREAD(4, 2, 4, false); break;
    default: SPREAD(5, 2, 3, false);
  }
#undef SPREAD
}

template <typename R>
int spread_t(bd_ctx* c, int k, const VecIn& v, size_t vr, R* grid) {
  const int np = (k + 1) / 2, K = c->pmeK, P = c->pme_p;
  // of the context's layouts the one with the least work for np pairs
  int l = 0;
  if (c->mesh_ng[1] && !sparse(c) &&
      layout_cost(np, c->mesh_ng[1], P) < layout_cost(np, c->mesh_ng[0], P))
    l = 1;
  const int ng = c->mesh_ng[l];
  SpreadArgs m;
  m.base = c->pme_base;
  m.w = c->pme_w;
  m.wx = c->pme_wx;
  m.ent = c->mesh_ent[l];
  m.bin = c->mesh_bin[l];
  m.K = K;
  m.npz = (K + kCols[ng][1] - 1) / kCols[ng][1];
  m.npatch = (int)patches(K, ng);
  m.nset = (np + ng - 1) / ng;
  m.nseg = segments(K, m.npatch * m.nset);
  m.np = np;
  m.N = c->N;
  m.vpk = c->pme_vpk;
  const bool planar = k == 1 ? c->pme_real1 : c->pme_planar;
  m.ps = planar ? 1 : 3;
  m.cs = planar ? (size_t)K * K * K : 1;
  c->launches++;
  k_mesh_pack<<<dim3(nblk(c->N, 128), np), 128, 0, c->stream>>>(
      v, vr, k, np, c->N, (typename GridVal<R>::T*)c->pme_vpk);
  const int nb = m.npatch * m.nseg * m.nset;
  c->launches++;
  switch (P) {
    case 4: launch_spread<4, R>(c, k, ng, nb, m, grid); break;
    case 6: launch_spread<6, R>(c, k, ng, nb, m, grid); break;
    default: launch_spread<8, R>(c, k, ng, nb, m, grid);
  }
  return BD_OK;
}

template <int P, typename R>
void launch_gather(bd_ctx* c, int k, const R* grid) {
  const dim3 g(nblk(c->N, 8), (k + 1) / 2);
#define GATHER(LAY_)                                                                      \
  k_mesh_gather<P, R, LAY_><<<g, 256, 0, c->stream>>>(c->pme_base, c->pme_w, (const R*)c->pme_wx, grid, c->N, c->pmeK, \
                                                      c->mesh_val)
  if (k == 1 && c->pme_real1)
    GATHER(kReal);
  else if (c->pme_planar)
    GATHER(kPlanar);
  else if (k == 1)
    GATHER(kSingle);
  else
    GATHER(kInterleaved);
#undef GATHER
}

template <typename R>
int gather_t(bd_ctx* c, int k, const R* grid) {
  c->launches++;
  switch (c->pme_p) {
    case 4: launch_gather<4, R>(c, k, grid); break;
    case 6: launch_gather<6, R>(c, k, grid); break;
    default: launch_gather<8, R>(c, k, grid);
  }
  return BD_OK;
}

}  // namespace

namespace bd {

int mesh_alloc(bd_ctx* c) {
  const int K = c->pmeK, N = c->N, P = c->pme_p, np = std::max(1, (c->nbk + 1) / 2);
  // a layout for single products and, where another does less work, one for
  // full blocks
  int best = 1;
  for (int ng = 2; ng <= 5; ng++)
    if (layout_cost(np, ng, P) < layout_cost(np, best, P)) best = ng;
  c->mesh_ng[0] = 1;
  c->mesh_ng[1] = best > 1 ? best : 0;
  size_t nbin_max = 0;
  int s;
  for (int l = 0; l < 2 && c->mesh_ng[l]; l++) {
    int ng = c->mesh_ng[l];
    size_t nbin = patches(K, ng) * K;
    size_t nent = (size_t)N * most_touched(K, P, kCols[ng][0]) * most_touched(K, P, kCols[ng][1]);
    s = alloc_all(c, {{&c->mesh_ent[l], 4 * nent}, {&c->mesh_bin[l], 4 * (nbin + 1)}});
    if (s != BD_OK) return s;
    nbin_max = std::max(nbin_max, nbin);
  }
  size_t nscan = nbin_max / kScanBlock + 1;
  return alloc_all(c, {{&c->mesh_sums, 4 * nscan},
                       {&c->mesh_cursor, 4 * nbin_max},
                       {&c->mesh_val, 48 * (size_t)N * np}});
}

void mesh_free(bd_ctx* c) {
  free_all({&c->mesh_ent[0], &c->mesh_ent[1], &c->mesh_bin[0], &c->mesh_bin[1], &c->mesh_sums,
            &c->mesh_cursor, &c->mesh_val});
}

static void scan_excl(bd_ctx* c, int* a, size_t n) {
  int nb = (int)((n + kScanBlock - 1) / kScanBlock);
  c->launches += 3;
  k_scan_sums<<<nb, 256, 0, c->stream>>>(a, n, c->mesh_sums);
  k_scan_blocks<<<1, 1024, 0, c->stream>>>(c->mesh_sums, nb, a + n);
  k_scan_place<<<nb, 256, 0, c->stream>>>(a, n, c->mesh_sums);
}

// The columns' bead lists for the base indices of the last k_pme_weights.
int mesh_prepare(bd_ctx* c) {
  const int N = c->N, P = c->pme_p, K = c->pmeK;
  for (int l = 0; l < 2 && c->mesh_ng[l]; l++) {
    const int CY = kCols[c->mesh_ng[l]][0], CZ = kCols[c->mesh_ng[l]][1], npz = (K + CZ - 1) / CZ;
    const size_t nbin = patches(K, c->mesh_ng[l]) * K;
    CU(cudaMemsetAsync(c->mesh_bin[l], 0, 4 * nbin, c->stream));
    CU(cudaMemsetAsync(c->mesh_cursor, 0, 4 * nbin, c->stream));
    c->launches += 3;
    k_mesh_list<<<nblk(N, 128), 128, 0, c->stream>>>(c->pme_base, N, K, P, CY, CZ, npz,
                                                     c->mesh_bin[l], nullptr, nullptr);
    scan_excl(c, c->mesh_bin[l], nbin);
    k_mesh_list<<<nblk(N, 128), 128, 0, c->stream>>>(c->pme_base, N, K, P, CY, CZ, npz,
                                                     c->mesh_cursor, c->mesh_bin[l],
                                                     c->mesh_ent[l]);
    k_mesh_sort<<<nblk((long long)nbin, 128), 128, 0, c->stream>>>(c->mesh_bin[l], nbin,
                                                                   c->mesh_ent[l]);
  }
  return launch_ok(c);
}

// grid = the spread of k right-hand sides v (component pointers, vr apart), as
// packed pairs.
int mesh_spread(bd_ctx* c, int k, const VecIn& v, size_t vr, void* grid) {
  return c->pme_f32 ? spread_t<float>(c, k, v, vr, (float*)grid)
                    : spread_t<double>(c, k, v, vr, (double*)grid);
}

// The pairs' interpolated values into mesh_val.
int mesh_gather(bd_ctx* c, int k, const void* grid) {
  return c->pme_f32 ? gather_t<float>(c, k, (const float*)grid)
                    : gather_t<double>(c, k, (const double*)grid);
}

}  // namespace bd
