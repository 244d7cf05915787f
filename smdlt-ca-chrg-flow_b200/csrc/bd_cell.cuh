// Periodic cell of the deforming lattice and cardinal B-splines, shared by
// the particle-mesh mobility (bd_pme.cu) and the Ewald Coulomb sum
// (bd_coulomb.cu).
#pragma once

#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "bd_ctx.cuh"

using namespace bd;

struct Cell {
  double H[9];     // lattice vectors as columns (lab frame), row-major 3x3
  double Hi[9];    // inverse
  double V;        // volume
};

static const int kMaxOrder = 8;

__device__ __forceinline__ void frac_of(const Cell& c, double x, double y, double z, double s[3]) {
  s[0] = c.Hi[0] * x + c.Hi[1] * y + c.Hi[2] * z;
  s[1] = c.Hi[3] * x + c.Hi[4] * y + c.Hi[5] * z;
  s[2] = c.Hi[6] * x + c.Hi[7] * y + c.Hi[8] * z;
}

// Cardinal B-spline weights: w[k] = M_p(f + k), k = 0..p-1, for the grid point
// floor(u) - k, from M_n(x) = (x M_{n-1}(x) + (n - x) M_{n-1}(x - 1))/(n - 1).
__device__ __forceinline__ void bspline(double f, int p, double* w) {
  double a[kMaxOrder], b[kMaxOrder];
  a[0] = f;
  a[1] = 1.0 - f;
  for (int n = 3; n <= p; n++) {
    for (int k = 0; k < n; k++) {
      double hi = k < n - 1 ? a[k] : 0.0, lo = k >= 1 ? a[k - 1] : 0.0;
      b[k] = ((f + k) * hi + (n - f - k) * lo) / (n - 1);
    }
    for (int k = 0; k < n; k++) a[k] = b[k];
  }
  for (int k = 0; k < p; k++) w[k] = a[k];
}

// bspline with the order known at compile time (loops unrolled, the
// recursion's arrays in registers).
template <int P>
__device__ __forceinline__ void bspline_t(double f, double* w) {
  double a[P], b[P];
  a[0] = f;
  a[1] = 1.0 - f;
#pragma unroll
  for (int n = 3; n <= P; n++) {
#pragma unroll
    for (int k = 0; k < n; k++) {
      double hi = k < n - 1 ? a[k] : 0.0, lo = k >= 1 ? a[k - 1] : 0.0;
      b[k] = ((f + k) * hi + (n - f - k) * lo) / (n - 1);
    }
#pragma unroll
    for (int k = 0; k < n; k++) a[k] = b[k];
  }
#pragma unroll
  for (int k = 0; k < P; k++) w[k] = a[k];
}

// The at most 27 neighbour cells of one cell as a single candidate list for a
// warp: lane l < ncell takes cell l's range, a warp scan of the counts places
// candidate m in the cell whose range holds it, so the lanes walk all cells
// at once (no chain of dependent loads per cell).  The arrays are the warp's
// own shared memory.
struct CandList {
  int start[32], excl[32], incl[32];

  // n cells per direction, cd the cell, cell_start the ranges; returns the
  // number of candidates (every lane)
  __device__ __forceinline__ int open(const int* n, const int* cd,
                                      const int* __restrict__ cell_start) {
    int lane = threadIdx.x & 31, lo[3], nd[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = n[d] >= 3 ? -1 : 0;
      nd[d] = n[d] >= 3 ? 3 : n[d];
    }
    int my_s = 0, my_n = 0;
    if (lane < nd[0] * nd[1] * nd[2]) {
      int a = lo[0] + lane / (nd[1] * nd[2]), b = lo[1] + (lane / nd[2]) % nd[1],
          c = lo[2] + lane % nd[2];
      int e0 = n[0] >= 3 ? (cd[0] + a + n[0]) % n[0] : a;
      int e1 = n[1] >= 3 ? (cd[1] + b + n[1]) % n[1] : b;
      int e2 = n[2] >= 3 ? (cd[2] + c + n[2]) % n[2] : c;
      int cc = (e0 * n[1] + e1) * n[2] + e2;
      my_s = cell_start[cc];
      my_n = cell_start[cc + 1] - my_s;
    }
    int in = my_n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, in, o);
      if (lane >= o) in += t;
    }
    __syncwarp();  // the previous list has been read
    start[lane] = my_s;
    excl[lane] = in - my_n;
    incl[lane] = in;
    __syncwarp();
    return __shfl_sync(0xffffffffu, in, 31);
  }

  // place of candidate m < total; cl is the lane's cursor, 0 before its first
  // candidate, candidates in increasing order
  __device__ __forceinline__ int at(int m, int& cl) const {
    while (m >= incl[cl]) cl++;  // ends at the last cell: m < total
    return start[cl] + (m - excl[cl]);
  }
};

// Minimum-image displacement; the cell is (b1, b2) in the xy plane and L e_z, and
// the nearest integer of |s| < 2^51 comes from adding and subtracting 1.5 2^52
// (two additions for one slow conversion).
struct Image {
  double h00, h01, h10, h11, g00, g01, g10, g11, Lz, iLz;
  __device__ __forceinline__ explicit Image(const Cell& c)
      : h00(c.H[0]), h01(c.H[1]), h10(c.H[3]), h11(c.H[4]), g00(c.Hi[0]), g01(c.Hi[1]),
        g10(c.Hi[3]), g11(c.Hi[4]), Lz(c.H[8]), iLz(c.Hi[8]) {}
  static __device__ __forceinline__ double nearest(double s) {
    return __dsub_rn(__dadd_rn(s, 6755399441055744.0), 6755399441055744.0);
  }
  __device__ __forceinline__ double operator()(const double4& pj, const double4& pi, double& dx,
                                               double& dy, double& dz) const {
    dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
    double n0 = nearest(g00 * dx + g01 * dy), n1 = nearest(g10 * dx + g11 * dy),
           n2 = nearest(iLz * dz);
    dx -= h00 * n0 + h01 * n1;
    dy -= h10 * n0 + h11 * n1;
    dz -= Lz * n2;
    return dx * dx + dy * dy + dz * dz;
  }
};

// Cell of a lab-frame position (0 for non-finite input).
__device__ __forceinline__ int cell_of_pos(const Cell& cell, const int* n, double x, double y,
                                           double z, int* cd) {
  double s[3];
  frac_of(cell, x, y, z, s);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double sd = s[d] - floor(s[d]);
    int c = (sd >= 0.0 && sd <= 1.0) ? (int)(sd * n[d]) : 0;
    cd[d] = c >= n[d] ? n[d] - 1 : c;
  }
  return (cd[0] * n[1] + cd[1]) * n[2] + cd[2];
}

static inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// Lab-frame cell of the current lattice: columns b1, b2, L e_z with (b1, b2)
// the Gauss-reduced basis of the lattice spanned by L1 and L2
// (|b1| <= |b2|, |b1.b2| <= |b1|^2/2).
static Cell make_cell(const Lat& l) {
  Cell c;
  double a[2] = {l.L1x, l.L1y}, b[2] = {l.L2x, l.L2y};
  for (int it = 0; it < 64; it++) {
    double aa = a[0] * a[0] + a[1] * a[1], bb = b[0] * b[0] + b[1] * b[1];
    if (aa > bb) {
      std::swap(a[0], b[0]);
      std::swap(a[1], b[1]);
      std::swap(aa, bb);
    }
    double mu = rint((a[0] * b[0] + a[1] * b[1]) / aa);
    if (mu == 0.0) break;
    b[0] -= mu * a[0];
    b[1] -= mu * a[1];
  }
  double H[9] = {a[0], b[0], 0.0, a[1], b[1], 0.0, 0.0, 0.0, l.L};
  memcpy(c.H, H, sizeof(H));
  double det = H[0] * (H[4] * H[8] - H[5] * H[7]) - H[1] * (H[3] * H[8] - H[5] * H[6]) +
               H[2] * (H[3] * H[7] - H[4] * H[6]);
  c.V = fabs(det);
  double* I = c.Hi;
  I[0] = (H[4] * H[8] - H[5] * H[7]) / det;
  I[1] = (H[2] * H[7] - H[1] * H[8]) / det;
  I[2] = (H[1] * H[5] - H[2] * H[4]) / det;
  I[3] = (H[5] * H[6] - H[3] * H[8]) / det;
  I[4] = (H[0] * H[8] - H[2] * H[6]) / det;
  I[5] = (H[2] * H[3] - H[0] * H[5]) / det;
  I[6] = (H[3] * H[7] - H[4] * H[6]) / det;
  I[7] = (H[1] * H[6] - H[0] * H[7]) / det;
  I[8] = (H[0] * H[4] - H[1] * H[3]) / det;
  return c;
}

// |b(m)|^2 = 1/|sum_{k=0}^{p-2} M_p(k+1) exp(2 pi i m k / K)|^2
static void bspline_moduli(int K, int p, double* out) {
  std::vector<double> Mk(p + 1, 0.0);
  // M_p at the integers 1..p-1 from the same recursion (f = 0)
  std::vector<double> a = {0.0, 1.0};
  for (int n = 3; n <= p; n++) {
    std::vector<double> b(n, 0.0);
    for (int k = 0; k < n; k++) {
      double hi = k < n - 1 ? a[k] : 0.0, lo = k >= 1 ? a[k - 1] : 0.0;
      b[k] = (k * hi + (n - k) * lo) / (n - 1);
    }
    a = b;
  }
  for (int m = 0; m < K; m++) {
    double re = 0, im = 0;
    for (int k = 0; k <= p - 2; k++) {
      double w = a[k + 1];  // M_p(k + 1)
      re += w * cos(2 * M_PI * m * k / K);
      im += w * sin(2 * M_PI * m * k / K);
    }
    double d = re * re + im * im;
    out[m] = d > 1e-300 ? 1.0 / d : 0.0;
  }
}

