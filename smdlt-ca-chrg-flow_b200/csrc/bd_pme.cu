// Matrix-free Rotne-Prager-Yamakawa mobility by smooth particle-mesh Ewald.
//
// No counterpart in the reference, whose mobility is a dense 3N x 3N matrix
// (calcHI, shear/src/main26.c:1530-1806).  It uses the same Beenakker Ewald
// split as calcHI, M = M_real + M_self + M_recip:
//  * M_real: for pairs closer than rc (lattice minimum image, rc below half
//    the narrowest cell width) the real-space Beenakker kernel with the
//    overlap form for r <= 2 (the C1..C4 terms of shear/src/main26.c:
//    1727-1741); the 3x3 pair tensors are built once per step into a row
//    list and applied as a sparse block product;
//  * M_self: 1 - 6 alpha/sqrt(pi) + 40 alpha^3/(3 sqrt(pi)) on the diagonal;
//  * M_recip = sum over k != 0 of (phi(k)/V)(I - k k^T/k^2) cos(k.r_ij),
//    phi(k) = (1 - k^2/3)(1 + k^2/4a^2 + k^4/8a^4)(6 pi/k^2) exp(-k^2/4a^2)
//    (the coefficient of shear/src/main26.c:1622), evaluated by smooth PME
//    (Essmann et al., J. Chem. Phys. 103, 8577 (1995)) on the deforming
//    cell: fractional coordinates s = H^-1 r, cardinal B-splines of even
//    order p on a K^3 grid, three-component R2C FFT, multiplication by
//    (phi/V)(I - k k^T/k^2) |b1 b2 b3|^2 with k = 2 pi H^-T m, C2R FFT and
//    interpolation with the same weights.
// The periodic lattice is described by its Gauss-reduced basis (shortest
// vectors of the lattice spanned by L1, L2 and L e_z): the lattice sums do
// not depend on the basis, and the reduced one keeps the grid spacing and the
// minimum-image cell widths bounded over the whole deformation period
// (|a| <= 1.16 L, widths >= 0.86 L for planar extension).
// Two conventions of calcHI are kept so that the sum reproduces its tensor:
//  * for overlapping beads (r < 2) its real-space form depends on the split
//    parameter; those pairs get that dependence at calcHI's own parameter
//    M_HI / rce (shear/src/main26.c:1536-1552) rather than at the PME one;
//  * calcHI stores only the diagonal entries of the self blocks
//    (shear/src/main26.c:1663-1700); the off-diagonal entries of the k-space
//    self sum, which a sheared or stretched cell makes non-zero, are removed.
// Spreading and interpolation are in bd_mesh.cu, the transforms in bd_fft.cuh
// (cuFFT for grid sizes it does not cover).  The spline weights, the columns' lists and the pair tensors are
// computed once per mobility build because its positions do not change during
// the Krylov solves.
#include <cufft.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "bd_ctx.cuh"
#include "bd_cell.cuh"
#include "bd_fft.cuh"
#include "bd_mesh.cuh"

using namespace bd;

#define CU(call) BD_CU(call)
#define CF(call) BD_CF(call)

// Per bead: base grid index floor(u) and the p weights in each lattice
// direction (u = K s, s wrapped into [0,1)).  Positions held in the rotated
// frame are taken to the lab frame with (cr, sr) = (cos, sin) of the lattice
// angle, x = x' cr - y' sr, y = x' sr + y' cr (inverseCoords,
// extensional/src/main14.c:1525-1535); lab-frame positions pass (1, 0).
template <typename R>
__global__ void k_pme_weights(Cell cell, const double* __restrict__ rx,
                              const double* __restrict__ ry, const double* __restrict__ rz,
                              double cr, double sr, int N, int K, int p, int* base, R* w,
                              double4* pos, int* err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double x = rx[i] * cr - ry[i] * sr, y = rx[i] * sr + ry[i] * cr, z = rz[i];
  pos[i] = make_double4(x, y, z, 0.0);
  double s[3];
  frac_of(cell, x, y, z, s);
  for (int d = 0; d < 3; d++) {
    double sd = s[d] - floor(s[d]);
    double u = sd * K;
    if (!(u >= 0.0 && u <= (double)K)) {  // non-finite position: keep indices in range
      u = 0.0;
      atomicOr(err, ERRB_NONFINITE);
    }
    int fl = (int)floor(u);
    double f = u - fl;
    if (fl >= K) fl -= K;
    base[3 * i + d] = fl;
    double wd[kMaxOrder];
    bspline(f, p, wd);
    for (int k = 0; k < p; k++) w[((size_t)3 * i + d) * kMaxOrder + k] = (R)wd[k];
  }
}

// Right-hand sides are packed in pairs: 2p and 2p + 1 are the real and
// imaginary parts of one complex grid of three components (the component
// fastest, pair p from 3 p K^3 on).  The influence tensor is real and even in
// k, so one complex transform, the multiplication and the inverse transform
// give both products, with no unpacking.  An odd last right-hand side, or a
// single one, has a zero imaginary part.

// The influence tensor on the full spectrum of the packed pairs, for grid sizes
// that go through cuFFT (thread per point and pair): points with m2 > K/2 take
// the tensor of their mirror -m, stored in the half spectrum.
template <typename R, typename Cx>
__global__ void k_pme_apply_influence(const R* __restrict__ infl, Cx* cgrid, int K, size_t np) {
  size_t K3 = (size_t)K * K * K;
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= K3 * np) return;
  size_t m = e % K3;
  int Kh = K / 2 + 1;
  int m0 = (int)(m / ((size_t)K * K)), m1 = (int)((m / K) % K), m2 = (int)(m % K);
  if (m2 > K / 2) {
    m0 = (K - m0) % K;
    m1 = (K - m1) % K;
    m2 = K - m2;
  }
  const R* t = infl + 6 * (((size_t)m0 * K + m1) * Kh + m2);
  Cx* b = cgrid + 3 * e;
  Cx x = b[0], y = b[1], z = b[2];
  Cx u, v, ww;
  u.x = t[0] * x.x + t[1] * y.x + t[2] * z.x;
  u.y = t[0] * x.y + t[1] * y.y + t[2] * z.y;
  v.x = t[1] * x.x + t[3] * y.x + t[4] * z.x;
  v.y = t[1] * x.y + t[3] * y.y + t[4] * z.y;
  ww.x = t[2] * x.x + t[4] * y.x + t[5] * z.x;
  ww.y = t[2] * x.y + t[4] * y.y + t[5] * z.y;
  b[0] = u;
  b[1] = v;
  b[2] = ww;
}

// Influence tensor on the half spectrum: (phi(k)/V)(I - k k^T/k^2) |b|^2,
// six components per point, zero at m = 0.
// Also the off-diagonal entries of sum_{k != 0} (phi/V)(I - k k^T/k^2) over
// the full spectrum (half spectrum with Hermitian multiplicity), one partial
// sum per block in soff_part[3 * block + (xy, xz, yz)].
template <typename R>
__global__ void __launch_bounds__(256) k_pme_influence(Cell cell, int K, double alpha,
                                                       const double* __restrict__ bsq, R* infl,
                                                       double* soff_part) {
  int Kh = K / 2 + 1;
  size_t n = (size_t)K * K * Kh;
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double sxy = 0, sxz = 0, syz = 0;
  __shared__ double red[3][256];
  if (e < n) {
    int m2 = (int)(e % Kh), m1 = (int)((e / Kh) % K), m0 = (int)(e / ((size_t)Kh * K));
    R* o = infl + 6 * e;
    if (m0 == 0 && m1 == 0 && m2 == 0) {
      for (int a = 0; a < 6; a++) o[a] = (R)0;
    } else {
      const double a2 = alpha * alpha;
      double t[6] = {0, 0, 0, 0, 0, 0}, k[3], kk = 0, phi = 0;
      auto add = [&](int n0, int n1, double share) {
        int s0 = n0 < (K + 1) / 2 ? n0 : n0 - K, s1 = n1 < (K + 1) / 2 ? n1 : n1 - K, s2 = m2;
        // k = 2 pi (s0 b0 + s1 b1 + s2 b2), b_d = row d of H^-1
        for (int a = 0; a < 3; a++)
          k[a] = 2.0 * M_PI *
                 (s0 * cell.Hi[0 * 3 + a] + s1 * cell.Hi[1 * 3 + a] + s2 * cell.Hi[2 * 3 + a]);
        kk = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
        phi = (1.0 - kk / 3.0) * (1.0 + kk / (4.0 * a2) + kk * kk / (8.0 * a2 * a2)) * 6.0 *
              M_PI / kk * exp(-kk / (4.0 * a2)) / cell.V;
        double f = share * phi * bsq[n0] * bsq[K + n1] * bsq[2 * K + m2];
        t[0] += f * (1.0 - k[0] * k[0] / kk);
        t[1] += f * (-k[0] * k[1] / kk);
        t[2] += f * (-k[0] * k[2] / kk);
        t[3] += f * (1.0 - k[1] * k[1] / kk);
        t[4] += f * (-k[1] * k[2] / kk);
        t[5] += f * (1.0 - k[2] * k[2] / kk);
      };
      // on the planes m2 = 0 and K/2 a point and its mirror are both stored:
      // their mean is even in k for the Nyquist indices of an even K too, so
      // the two right-hand sides of a pair do not mix
      bool both = m2 == 0 || 2 * m2 == K;
      if (both) add((K - m0) % K, (K - m1) % K, 0.5);
      add(m0, m1, both ? 0.5 : 1.0);
      for (int a = 0; a < 6; a++) o[a] = (R)t[a];
      double mult = (m2 == 0 || (K % 2 == 0 && m2 == K / 2)) ? 1.0 : 2.0;
      sxy = -mult * phi * k[0] * k[1] / kk;
      sxz = -mult * phi * k[0] * k[2] / kk;
      syz = -mult * phi * k[1] * k[2] / kk;
    }
  }
  red[0][threadIdx.x] = sxy;
  red[1][threadIdx.x] = sxz;
  red[2][threadIdx.x] = syz;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
      for (int a = 0; a < 3; a++) red[a][threadIdx.x] += red[a][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 3) soff_part[3 * blockIdx.x + threadIdx.x] = red[threadIdx.x][0];
}

// Fixed-order sum of the per-block self off-diagonal partials.
__global__ void k_pme_soff_fin(const double* __restrict__ part, int nb, double* soff) {
  __shared__ double red[3][256];
  double a0 = 0, a1 = 0, a2 = 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    a0 += part[3 * b];
    a1 += part[3 * b + 1];
    a2 += part[3 * b + 2];
  }
  red[0][threadIdx.x] = a0;
  red[1][threadIdx.x] = a1;
  red[2][threadIdx.x] = a2;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
      for (int a = 0; a < 3; a++) red[a][threadIdx.x] += red[a][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 3) soff[threadIdx.x] = red[threadIdx.x][0];
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

// Self part and the interpolated value of component c, right-hand side r, bead
// i: mesh + self v - (S_off v)_c.
__device__ __forceinline__ double with_self(double mesh, int c, double self,
                                            const double* __restrict__ soff, const VecIn& v,
                                            size_t o) {
  double v0 = v.p[0][o], v1 = v.p[1][o], v2 = v.p[2][o];
  double sxy = soff[0], sxz = soff[1], syz = soff[2];
  if (c == 0) return mesh + self * v0 - sxy * v1 - sxz * v2;
  if (c == 1) return mesh + self * v1 - sxy * v0 - syz * v2;
  return mesh + self * v2 - sxz * v0 - syz * v1;
}

// What the last kernel of a product adds to its real-space sums and where it
// writes them.
struct Finish {
  const double* val;  // the interpolated values, 6 per bead and pair
  int N;
  double self;
  const double* soff;
  VecIn v;
  size_t vr;
  double* o[3];
  int ostride;
  size_t orr;
  int k;

  // value e = 3 h + c of packed pair pr, real-space sum x
  __device__ __forceinline__ void write(double x, int pr, int e, int i) const {
    int r = 2 * pr + e / 3, c = e % 3;
    if (r >= k) return;
    double mesh = x + val[((size_t)pr * N + i) * 6 + e];
    double* dst = c == 0 ? o[0] : c == 1 ? o[1] : o[2];
    dst[(size_t)r * orr + (size_t)i * ostride] =
        with_self(mesh, c, self, soff, v, (size_t)r * vr + (size_t)i * v.stride);
  }
};

// The real-space sums from (t1, t2 / r^2) per pair, the minimum image formed
// here, FP64 sums (FP64 contexts, and FP32 ones without the stored (t1, w)),
// and the rest of the product, for packed pair blockIdx.y.  One warp per bead, lanes over the pair row,
// a butterfly, lane e < 6 writes value e.
template <typename R>
__global__ void __launch_bounds__(256)
    k_pme_real_rows(int N, const int* __restrict__ rcnt, const int* __restrict__ rrows,
                    const double4* __restrict__ pos, Cell cell, const R* __restrict__ tt, int rcap,
                    Finish fin) {
  constexpr int KG = 2, NA = 3 * KG;
  int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= N) return;
  const VecIn& v = fin.v;
  int r0 = KG * blockIdx.y, kc = min(KG, fin.k - r0);
  double u[NA];
#pragma unroll
  for (int e = 0; e < NA; e++) u[e] = 0.0;
  int n = rcnt[i];
  const int* prow = rrows + (size_t)i * rcap;
  // the cell is (b1, b2) in the xy plane and L e_z: a 2 x 2 block and L
  double4 pi = pos[i];
  const double h00 = cell.H[0], h01 = cell.H[1], h10 = cell.H[3], h11 = cell.H[4];
  const double g00 = cell.Hi[0], g01 = cell.Hi[1], g10 = cell.Hi[3], g11 = cell.Hi[4];
  const double Lz = cell.H[8], iLz = cell.Hi[8];
  for (int kk = lane; kk < n; kk += 32) {
    int j = prow[kk];
    double4 pj = pos[j];
    double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    double s0 = g00 * dx + g01 * dy, s1 = g10 * dx + g11 * dy, s2 = iLz * dz;
    s0 -= rint(s0);
    s1 -= rint(s1);
    s2 -= rint(s2);
    dx = h00 * s0 + h01 * s1;
    dy = h10 * s0 + h11 * s1;
    dz = Lz * s2;
    const R* tk = tt + 2 * ((size_t)i * rcap + kk);
    double t1 = tk[0], t2r = tk[1];  // t1 and t2 / r^2 of the pair
#pragma unroll
    for (int r = 0; r < KG; r++) {
      if (r >= kc) break;
      size_t o = (size_t)(r0 + r) * fin.vr + (size_t)j * v.stride;
      double x0 = v.p[0][o], x1 = v.p[1][o], x2 = v.p[2][o];
      double qq = t2r * (dx * x0 + dy * x1 + dz * x2);
      u[3 * r] += t1 * x0 + qq * dx;
      u[3 * r + 1] += t1 * x1 + qq * dy;
      u[3 * r + 2] += t1 * x2 + qq * dz;
    }
  }
#pragma unroll
  for (int e = 0; e < NA; e++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u[e] += __shfl_xor_sync(0xffffffffu, u[e], o);
  double mine = 0.0;
#pragma unroll
  for (int e = 0; e < NA; e++)
    if (e == lane) mine = u[e];
  if (lane < NA) fin.write(mine, blockIdx.y, lane, i);
}

// The real-space part of a block product and the rest of it (FP32 block
// products): for every packed pair p0 + p and bead i, sum_j (T_ij v_j)_c of the
// pair's vector h (0: real part, 1: imaginary part), for NP pairs (at most
// five) in one pass over the pair rows.  One warp per bead; a lane takes
// row entries, each an index and the preparation's float4 (t1, w): T_ij =
// t1 I + s w w^T, the sign s of t2 kept in the lowest mantissa bit of t1;
// then it reads the neighbour's six inputs of every pair (the packed record
// vpk[(p N + j) 8], a float4 and a float2) and adds T_ij v into 6 NP FP32
// partial sums (a lane sums about a 32nd of the row).  The
// partials are summed over the warp by a transposing butterfly (31 exchanges
// per 32 values, lane l ends with the sum of value l), its first two stages
// in FP32 and the last three in FP64.
template <int NP>
__global__ void __launch_bounds__(256, 3) k_pme_real_pairs(
    const int* __restrict__ rcnt, const int* __restrict__ rrows, const float4* __restrict__ rw,
    int rcap, const float* __restrict__ vpk, int N, int p0, Finish fin) {
  constexpr int NV = 6 * NP;
  int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= N) return;
  float u[NV];
#pragma unroll
  for (int e = 0; e < NV; e++) u[e] = 0.f;
  int n = rcnt[i];
  const int* prow = rrows + (size_t)i * rcap;
  const float4* prw = rw + (size_t)i * rcap;
  for (int kk = lane; kk < n; kk += 32) {
    int j = __ldg(prow + kk);
    float4 q = __ldg(prw + kk);
    float s = (__float_as_uint(q.x) & 1u) ? -1.f : 1.f;
#pragma unroll
    for (int p = 0; p < NP; p++) {
      const float4* vj = (const float4*)(vpk + ((size_t)(p0 + p) * N + j) * 8);
      float4 a = __ldg(vj);
      float2 b = __ldg((const float2*)(vj + 1));
      float qa = s * (q.y * a.x + q.z * a.y + q.w * a.z);
      float qb = s * (q.y * a.w + q.z * b.x + q.w * b.y);
      u[6 * p] += q.x * a.x + qa * q.y;
      u[6 * p + 1] += q.x * a.y + qa * q.z;
      u[6 * p + 2] += q.x * a.z + qa * q.w;
      u[6 * p + 3] += q.x * a.w + qb * q.y;
      u[6 * p + 4] += q.x * b.x + qb * q.z;
      u[6 * p + 5] += q.x * b.y + qb * q.w;
    }
  }
  // the first two exchanges in FP32 (sums of 2 and 4 lanes), the rest in FP64
  float f[32];
#pragma unroll
  for (int e = 0; e < 32; e++) f[e] = e < NV ? u[e] : 0.f;
#pragma unroll
  for (int off = 16; off >= 8; off >>= 1) {
    bool up = lane & off;
#pragma unroll
    for (int e = 0; e < off; e++) {
      float send = up ? f[e] : f[e + off];
      float keep = up ? f[e + off] : f[e];
      f[e] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  double d[8];
#pragma unroll
  for (int e = 0; e < 8; e++) d[e] = (double)f[e];
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) {
    bool up = lane & off;
#pragma unroll
    for (int e = 0; e < off; e++) {
      double send = up ? d[e] : d[e + off];
      double keep = up ? d[e + off] : d[e];
      d[e] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  // value 6 p + 3 h + c
  if (lane < NV) fin.write(d[0], p0 + lane / 6, lane % 6, i);
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

// Positions in cell order, the bead index in the fourth component: the row
// build streams a cell's beads with one contiguous load each.
__global__ void k_rl_fill(const int* __restrict__ cell_of, const int* __restrict__ cell_start,
                          int* cursor, const double4* __restrict__ pos, double4* spos, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int c = cell_of[i];
  double4 p = pos[i];
  p.w = __longlong_as_double((long long)i);
  spos[cell_start[c] + atomicAdd(&cursor[c], 1)] = p;
}

// Pairs within rc (lattice minimum image): rows of bead indices and, per
// pair, the stored tensor: (t1, w) where the products read it (rw, FP32 block
// contexts), else t1 and t2 / r^2.
// One warp per bead.  The at most 27 neighbour cells form one candidate list
// (lane l takes cell l's range, a warp scan places candidate m); the lanes
// test 32 candidates at a time and queue the hits in shared memory, and the
// pair terms (erfc, exp: most of the FP64 work, needed by about one candidate
// in eight) are formed 32 queued pairs at a time, so no lane idles in them
// and the row's stores are contiguous.  Overlapping pairs, whose terms cost
// three times as much, have a queue of their own.  Bound by the FP64 pipe:
// 193 M tests and 24 M pair terms at 50 000 beads, cutoff 14.5.  A thread per
// bead, with its stores a row apart, took 6.01 ms there; this takes 1.33 ms.
template <typename R>
__global__ void __launch_bounds__(256, 3)
    k_rl_rows(Cell cell, RGeom g, const double4* __restrict__ pos, int N,
              const int* __restrict__ cell_start, const double4* __restrict__ spos, double rc2,
              double alpha, double alpha_ref, int rcap, int* cnt, int* rows, R* tt, float4* rw,
              int* need, int* err) {
  __shared__ CandList c_list[8];
  __shared__ int c_queue[8][2][64];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + wl;
  if (i >= N) return;
  const double4 p = pos[i];
  int cd[3];
  cell_of_pos(cell, g.n, p.x, p.y, p.z, cd);
  const int total = c_list[wl].open(g.n, cd, cell_start);
  // displacement to a bead, minimum image; the cell is (b1, b2) in the xy
  // plane and L e_z, and the nearest integer of |s| < 2^51 comes from adding
  // and subtracting 1.5 2^52 (two additions for one slow conversion)
  const double h00 = cell.H[0], h01 = cell.H[1], h10 = cell.H[3], h11 = cell.H[4];
  const double g00 = cell.Hi[0], g01 = cell.Hi[1], g10 = cell.Hi[3], g11 = cell.Hi[4];
  const double Lz = cell.H[8], iLz = cell.Hi[8];
  auto nearest = [](double s) {
    return __dsub_rn(__dadd_rn(s, 6755399441055744.0), 6755399441055744.0);
  };
  auto image = [&](const double4& pj, double& dx, double& dy, double& dz) {
    dx = pj.x - p.x, dy = pj.y - p.y, dz = pj.z - p.z;
    double n0 = nearest(g00 * dx + g01 * dy), n1 = nearest(g10 * dx + g11 * dy),
           n2 = nearest(iLz * dz);
    dx -= h00 * n0 + h01 * n1;
    dy -= h10 * n0 + h11 * n1;
    dz -= Lz * n2;
    return dx * dx + dy * dy + dz * dz;
  };
  // pair terms of the first nq pairs of a queue into the row from entry n on
  auto emit = [&](auto overlap, int n, int nq) {
    constexpr bool OV = decltype(overlap)::value;
    if (lane >= nq || n + lane >= rcap) return;
    double4 pj = spos[c_queue[wl][OV][lane]];
    int j = (int)__double_as_longlong(pj.w);
    double dx, dy, dz, t1, t2, rr = image(pj, dx, dy, dz);
    double r = sqrt(rr), ir = 1.0 / r, irr = ir * ir;
    pair_terms<OV>(alpha, alpha_ref, rr, r, ir, irr, t1, t2);
    size_t e = (size_t)i * rcap + n + lane;
    rows[e] = j;
    if (rw) {
      double sw = sqrt(fabs(t2)) * ir;
      unsigned b = (__float_as_uint((float)t1) & ~1u) | (t2 < 0.0 ? 1u : 0u);
      rw[e] = make_float4(__uint_as_float(b), (float)(sw * dx), (float)(sw * dy),
                          (float)(sw * dz));
    } else {
      tt[2 * e] = (R)t1;
      tt[2 * e + 1] = (R)(t2 * irr);
    }
  };
  int n = 0, nq0 = 0, nq1 = 0, cl = 0;
  // appends the hits of one kind to their queue; a full batch goes to the row
  auto push = [&](auto overlap, bool in, int j, int& nq) {
    constexpr bool OV = decltype(overlap)::value;
    unsigned hit = __ballot_sync(0xffffffffu, in);
    if (hit == 0) return;
    int* queue = c_queue[wl][OV];
    if (in) queue[nq + __popc(hit & ((1u << lane) - 1u))] = j;
    nq += __popc(hit);
    __syncwarp();
    if (nq >= 32) {
      emit(overlap, n, 32);
      n += 32;
      nq -= 32;
      __syncwarp();
      int rest = lane < nq ? queue[32 + lane] : 0;
      __syncwarp();
      if (lane < nq) queue[lane] = rest;
      __syncwarp();
    }
  };
  // the next candidate's load is in flight while this one is tested
  int at = -1, next_at = -1;
  double4 pj = p, next = p;
  auto fetch = [&](int m) {
    next_at = -1;
    if (m < total) {
      next_at = c_list[wl].at(m, cl);
      next = spos[next_at];
    }
  };
  fetch(lane);
  for (int m0 = 0; m0 < total; m0 += 32) {
    at = next_at;
    pj = next;
    fetch(m0 + 32 + lane);
    double dx, dy, dz, rr = image(pj, dx, dy, dz);
    bool in = at >= 0 && !(rr >= rc2) && (int)__double_as_longlong(pj.w) != i;
    bool near = rr < 4.0;
    push(std::integral_constant<bool, false>(), in && !near, at, nq0);
    push(std::integral_constant<bool, true>(), in && near, at, nq1);
  }
  emit(std::integral_constant<bool, false>(), n, nq0);
  n += nq0;
  emit(std::integral_constant<bool, true>(), n, nq1);
  n += nq1;
  if (lane == 0) {
    cnt[i] = min(n, rcap);
    if (n > rcap) {
      if (need)
        atomicMax(need, n);  // the host grows the rows and builds them again
      else
        atomicOr(err, ERRB_NBR_OVERFLOW);
    }
  }
}

namespace bd {

int pme_alloc(bd_ctx* c) {
  if (c->pme_grid) return BD_OK;
  int K = c->pmeK, N = c->N;
  size_t K3 = (size_t)K * K * K, Ks = (size_t)K * K * (K / 2 + 1);
  c->pme_f32 = c->p.precision == BD_PREC_FP32;
  size_t es = c->pme_f32 ? 4 : 8;  // grid, spectrum, influence and pair tensors
  // the packed pairs' grids for the largest number of right-hand sides
  size_t nr = (size_t)std::max(1, c->nbk);
  size_t grid_bytes = 2 * es * 3 * K3 * ((nr + 1) / 2);
  CU(cudaMalloc(&c->pme_grid, grid_bytes));
  CU(cudaMalloc(&c->pme_tw, 2 * es * K));
  CU(cudaMalloc(&c->pme_infl, es * 6 * Ks));
  CU(cudaMalloc(&c->pme_bsq, 8 * 3 * (size_t)K));
  c->pme_nblk = (int)((Ks + 255) / 256);
  CU(cudaMalloc(&c->pme_soff, 8 * (3 * (size_t)c->pme_nblk + 3)));
  CU(cudaMalloc(&c->pme_base, 4 * 3 * (size_t)N));
  CU(cudaMalloc(&c->pme_w, es * 3 * (size_t)N * kMaxOrder));
  // default row cap: 2.5 times the mean number of beads within the cutoff at
  // the system's density, at least 512, a multiple of 32
  if (c->p.pme_max_pairs > 0) {
    c->rl_cap = c->p.pme_max_pairs;
  } else {
    double mean = 4.0 / 3.0 * M_PI * c->pme_rc * c->pme_rc * c->pme_rc * N / c->boxvol;
    c->rl_cap = std::max(512, ((int)ceil(2.5 * mean) + 31) / 32 * 32);
  }
  CU(cudaMalloc(&c->rl_cnt, 4 * (size_t)N));
  CU(cudaMalloc(&c->rl_need, 4));
  CU(cudaMemsetAsync(c->rl_need, 0, 4, c->stream));
  CU(cudaMalloc(&c->rl_rows, 4 * (size_t)N * c->rl_cap));
  CU(cudaMalloc(&c->rl_pos, 32 * (size_t)N));
  if (c->pme_f32 && nr > 1) {
    CU(cudaMalloc(&c->pme_vpk, 32 * (size_t)N * ((nr + 1) / 2)));
    CU(cudaMalloc(&c->rl_w, 16 * (size_t)N * c->rl_cap));
    c->bytes += 32 * (size_t)N * ((nr + 1) / 2) + 16 * (size_t)N * c->rl_cap;
  } else {  // the products of contexts with rl_w read the pair tensors there
    CU(cudaMalloc(&c->rl_tt, 2 * es * (size_t)N * c->rl_cap));
    c->bytes += 2 * es * (size_t)N * c->rl_cap;
  }
  c->rl_ncell_cap = 4096;
  CU(cudaMalloc(&c->rl_cell_of, 4 * (size_t)N));
  CU(cudaMalloc(&c->rl_spos, 32 * (size_t)N));
  CU(cudaMalloc(&c->rl_cell_count, 4 * (size_t)c->rl_ncell_cap));
  CU(cudaMalloc(&c->rl_cell_start, 4 * (size_t)(c->rl_ncell_cap + 1)));
  CU(cudaMalloc(&c->rl_cursor, 4 * (size_t)c->rl_ncell_cap));
  CU(cudaMemsetAsync(c->rl_cell_count, 0, 4 * (size_t)c->rl_ncell_cap, c->stream));
  c->bytes += grid_bytes + es * 6 * Ks + (24 + 2 * es) * (size_t)K + 12 * (size_t)N +
              3 * es * (size_t)N * kMaxOrder + 4 * (size_t)N + (size_t)N * c->rl_cap * 4 + 32 * (size_t)N +
              36 * (size_t)N + 12 * (size_t)c->rl_ncell_cap;
  if (!fft_has_size(K)) {
    // one pair's three interleaved components, in place
    int n[3] = {K, K, K};
    cufftHandle f;
    CF(cufftPlanMany(&f, 3, n, n, 3, 1, n, 3, 1, c->pme_f32 ? CUFFT_C2C : CUFFT_Z2Z, 3));
    CF(cufftSetStream(f, c->stream));
    c->pme_plan = (int)f + 1;
  }
  std::vector<double> tw(2 * (size_t)K);
  std::vector<float> tw32(2 * (size_t)K);
  for (int m = 0; m < K; m++) {
    tw[2 * m] = cos(2.0 * M_PI * m / K);
    tw[2 * m + 1] = -sin(2.0 * M_PI * m / K);
    tw32[2 * m] = (float)tw[2 * m];
    tw32[2 * m + 1] = (float)tw[2 * m + 1];
  }
  CU(cudaMemcpyAsync(c->pme_tw, c->pme_f32 ? (const void*)tw32.data() : (const void*)tw.data(),
                     2 * es * K, cudaMemcpyHostToDevice, c->stream));
  std::vector<double> bs(3 * (size_t)K);
  bspline_moduli(K, c->pme_p, bs.data());
  for (int d = 1; d < 3; d++)
    for (int m = 0; m < K; m++) bs[(size_t)d * K + m] = bs[m];
  CU(cudaMemcpyAsync(c->pme_bsq, bs.data(), 8 * bs.size(), cudaMemcpyHostToDevice, c->stream));
  CU(cudaStreamSynchronize(c->stream));
  return BD_OK;
}

void pme_free(bd_ctx* c) {
  if (c->pme_plan) cufftDestroy((cufftHandle)(c->pme_plan - 1));
  mesh_free(c);
  void* ptrs[] = {c->pme_vpk, c->rl_w, c->rl_need, c->pme_grid, c->pme_tw, c->pme_infl, c->pme_bsq, c->pme_soff, c->pme_base, c->pme_w,
                  c->rl_cnt, c->rl_rows, c->rl_pos, c->rl_tt, c->rl_cell_of, c->rl_spos, c->rl_cell_count,
                  c->rl_cell_start, c->rl_cursor};
  for (void* q : ptrs)
    if (q) cudaFree(q);
}

// Preparation for the current positions, in the frame calcHI reads them
// (extension: rotated by the lattice angle, taken to the lab frame here):
// spline weights, influence tensor of the current cell, self off-diagonal
// sums, real-space pair list and tensors.  The products that follow use this
// configuration until the next preparation, as the dense matrix does.
// Pair rows of a larger cap (the rows are rebuilt by the caller).
static int rl_grow(bd_ctx* c, int cap) {
  size_t N = c->N, es = c->pme_f32 ? 4 : 8, old = (size_t)c->rl_cap;
  CU(cudaStreamSynchronize(c->stream));
  cudaFree(c->rl_rows);
  c->rl_rows = nullptr;
  CU(cudaMalloc(&c->rl_rows, 4 * N * cap));
  c->bytes += 4 * N * (cap - old);
  if (c->rl_tt) {
    cudaFree(c->rl_tt);
    c->rl_tt = nullptr;
    CU(cudaMalloc(&c->rl_tt, 2 * es * N * cap));
    c->bytes += 2 * es * N * (cap - old);
  }
  if (c->rl_w) {
    cudaFree(c->rl_w);
    c->rl_w = nullptr;
    CU(cudaMalloc(&c->rl_w, 16 * N * cap));
    c->bytes += 16 * N * (cap - old);
  }
  c->rl_cap = cap;
  CU(cudaMemsetAsync(c->rl_need, 0, 4, c->stream));
  return BD_OK;
}

int pme_prepare(bd_ctx* c, const Lat& l) {
  int s;
  if ((s = pme_alloc(c)) != BD_OK) return s;
  Cell cell = make_cell(l);
  double cr = 1.0, sr = 0.0;
  if (l.flow == BD_FLOW_EXT) {
    cr = l.cth;
    sr = l.sth;
  }
  double rc = c->pme_rc, alpha = c->pme_alpha;
  int K = c->pmeK, N = c->N;
  // calcHI's split parameter at this step, for its overlap convention
  double rce = l.treal <= c->tp / 2 ? l.L2yp : 2.0 * l.L2yp;
  double alpha_ref = 4.0 / rce;
  c->launches += 3;
  if (c->pme_f32)
    k_pme_weights<float><<<nblk(N, 128), 128, 0, c->stream>>>(
        cell, c->rx, c->ry, c->rz, cr, sr, N, K, c->pme_p, c->pme_base, (float*)c->pme_w,
        (double4*)c->rl_pos, c->err);
  else
    k_pme_weights<double><<<nblk(N, 128), 128, 0, c->stream>>>(
        cell, c->rx, c->ry, c->rz, cr, sr, N, K, c->pme_p, c->pme_base, (double*)c->pme_w,
        (double4*)c->rl_pos, c->err);
  if ((s = mesh_prepare(c)) != BD_OK) return s;
  if (c->pme_f32)
    k_pme_influence<float><<<c->pme_nblk, 256, 0, c->stream>>>(
        cell, K, alpha, c->pme_bsq, (float*)c->pme_infl, c->pme_soff + 3);
  else
    k_pme_influence<double><<<c->pme_nblk, 256, 0, c->stream>>>(
        cell, K, alpha, c->pme_bsq, (double*)c->pme_infl, c->pme_soff + 3);
  k_pme_soff_fin<<<1, 256, 0, c->stream>>>(c->pme_soff + 3, c->pme_nblk, c->pme_soff);
  if ((s = launch_ok(c)) != BD_OK) return s;
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
                                                 (const double4*)c->rl_pos,
                                                 (double4*)c->rl_spos, N);
  if ((s = launch_ok(c)) != BD_OK) return s;
  // the pair rows; with the default cap (no pme_max_pairs), rows that
  // overflow it are grown to 1.25 times the longest row and built again
  int* need = c->p.pme_max_pairs > 0 ? nullptr : c->rl_need;
  for (int pass = 0; pass < 2; pass++) {
    if (c->pme_f32)
      k_rl_rows<float><<<nblk(N, 8), 256, 0, c->stream>>>(
          cell, g, (const double4*)c->rl_pos, N, c->rl_cell_start, (const double4*)c->rl_spos,
          rc * rc, alpha,
          alpha_ref, c->rl_cap, c->rl_cnt, c->rl_rows, (float*)c->rl_tt, c->rl_w, need, c->err);
    else
      k_rl_rows<double><<<nblk(N, 8), 256, 0, c->stream>>>(
          cell, g, (const double4*)c->rl_pos, N, c->rl_cell_start, (const double4*)c->rl_spos,
          rc * rc, alpha,
          alpha_ref, c->rl_cap, c->rl_cnt, c->rl_rows, (double*)c->rl_tt, nullptr, need, c->err);
    if (!need) break;
    int longest = 0;
    CU(cudaMemcpyAsync(&longest, need, 4, cudaMemcpyDeviceToHost, c->stream));
    if ((s = check(c)) != BD_OK) return s;
    if (longest <= c->rl_cap) break;
    if ((s = rl_grow(c, ((int)ceil(1.25 * longest) + 31) / 32 * 32)) != BD_OK) return s;
  }
  // the cell and calcHI's split parameter of this configuration, for the
  // products until the next preparation
  memcpy(c->pme_cellbuf, cell.H, sizeof(cell.H));
  memcpy(c->pme_cellbuf + 9, cell.Hi, sizeof(cell.Hi));
  c->pme_cellbuf[18] = cell.V;
  c->pme_alpha_ref = alpha_ref;
  double a = alpha;
  c->pme_self = 1.0 - 6.0 / sqrt(M_PI) * a + 40.0 / (3.0 * sqrt(M_PI)) * a * a * a;
  c->Dtr[0] = c->Dtr[1] = c->Dtr[2] = c->pme_self;
  c->pme_ready = true;
  c->hi_built = true;
  return launch_ok(c);
}

// out_r = M v_r by PME for k right-hand sides given by component pointers
// (VecIn) and RHS strides vr (input) and orr (output).
template <typename R, typename Cx>
static int pme_apply_t(bd_ctx* c, int k, const VecIn& v, size_t vr, double* o0, double* o1,
                       double* o2, int ostride, size_t orr) {
  int K = c->pmeK, N = c->N, s;
  size_t K3 = (size_t)K * K * K;
  if (k < 1 || k > std::max(1, c->nbk)) return BD_ERR_ARG;
  int nb8 = nblk(N, 8), np = (k + 1) / 2;
  Cx* g = (Cx*)c->pme_grid;
  if ((s = mesh_spread(c, k, v, vr, g)) != BD_OK) return s;
  if (!c->pme_plan) {
    s = sizeof(R) == 4 ? fft_influence_f32(c, K, g, np, c->pme_infl, c->pme_tw)
                       : fft_influence_f64(c, K, g, np, c->pme_infl, c->pme_tw);
    if (s != BD_OK) return s;
  } else {
    for (int dir : {CUFFT_FORWARD, CUFFT_INVERSE}) {
      for (int p = 0; p < np; p++) {
        Cx* gp = g + 3 * K3 * p;
        if constexpr (sizeof(R) == 4)
          CF(cufftExecC2C((cufftHandle)(c->pme_plan - 1), (cufftComplex*)gp, (cufftComplex*)gp, dir));
        else
          CF(cufftExecZ2Z((cufftHandle)(c->pme_plan - 1), (cufftDoubleComplex*)gp,
                          (cufftDoubleComplex*)gp, dir));
      }
      if (dir == CUFFT_FORWARD) {
        c->launches++;
        k_pme_apply_influence<R, Cx><<<nblk((long long)K3 * np, 256), 256, 0, c->stream>>>(
            (const R*)c->pme_infl, g, K, (size_t)np);
      }
    }
  }
  if ((s = mesh_gather(c, k, g)) != BD_OK) return s;
  Finish fin;
  fin.val = c->mesh_val;
  fin.N = N;
  fin.self = c->pme_self;
  fin.soff = c->pme_soff;
  fin.v = v;
  fin.vr = vr;
  fin.o[0] = o0;
  fin.o[1] = o1;
  fin.o[2] = o2;
  fin.ostride = ostride;
  fin.orr = orr;
  fin.k = k;
  if constexpr (sizeof(R) == 4) {
    // FP32 contexts with the stored (t1, w): passes over the rows of up to five
    // pairs (30 FP32 partial sums per lane at 80 registers)
    if (c->rl_w) {
      for (int p0 = 0; p0 < np; p0 += 5) {
        c->launches++;
#define PME_REAL(NP_)                                                                        \
  k_pme_real_pairs<NP_><<<nb8, 256, 0, c->stream>>>(c->rl_cnt, c->rl_rows, c->rl_w, c->rl_cap, \
                                                    c->pme_vpk, N, p0, fin)
        switch (std::min(5, np - p0)) {
          case 1: PME_REAL(1); break;
          case 2: PME_REAL(2); break;
          case 3: PME_REAL(3); break;
          case 4: PME_REAL(4); break;
          default: PME_REAL(5);
        }
#undef PME_REAL
      }
      return BD_OK;
    }
  }
  Cell cell;
  memcpy(cell.H, c->pme_cellbuf, sizeof(cell.H));
  memcpy(cell.Hi, c->pme_cellbuf + 9, sizeof(cell.Hi));
  cell.V = c->pme_cellbuf[18];
  c->launches++;
  k_pme_real_rows<R><<<dim3(nb8, np), 256, 0, c->stream>>>(
      N, c->rl_cnt, c->rl_rows, (const double4*)c->rl_pos, cell, (const R*)c->rl_tt, c->rl_cap,
      fin);
  return BD_OK;
}

static int pme_apply_k(bd_ctx* c, int k, const VecIn& v, size_t vr, double* o0, double* o1,
                       double* o2, int ostride, size_t orr) {
  if (!c->pme_ready) return BD_ERR_STATE;
  prof_begin(c, BD_PROF_MATVEC);
  int s = c->pme_f32
              ? pme_apply_t<float, cufftComplex>(c, k, v, vr, o0, o1, o2, ostride, orr)
              : pme_apply_t<double, cufftDoubleComplex>(c, k, v, vr, o0, o1, o2, ostride, orr);
  prof_end(c, BD_PROF_MATVEC);
  if (s != BD_OK) return s;
  return launch_ok(c);
}

int pme_apply(bd_ctx* c, const VecIn& v, double* o0, double* o1, double* o2, int ostride) {
  return pme_apply_k(c, 1, v, 0, o0, o1, o2, ostride, 0);
}

int pme_apply_multi(bd_ctx* c, int k, const double* X, size_t xs, double* Y, size_t ys) {
  int NTp = c->NT * 32;
  VecIn v = {{X, X + NTp, X + 2 * (size_t)NTp}, 1};
  return pme_apply_k(c, k, v, xs, Y, Y + NTp, Y + 2 * (size_t)NTp, 1, ys);
}

}  // namespace bd
