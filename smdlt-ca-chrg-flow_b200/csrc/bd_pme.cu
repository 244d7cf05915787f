// Matrix-free Rotne-Prager-Yamakawa mobility by smooth particle-mesh Ewald.
//
// No counterpart in the reference, whose mobility is a dense 3N x 3N matrix
// (calcHI, shear/src/main26.c:1530-1806).  It uses the same Beenakker Ewald
// split as calcHI, M = M_real + M_self + M_recip:
//  * M_real: for pairs closer than rc (lattice minimum image, rc below half
//    the narrowest cell width) the real-space Beenakker kernel with the
//    overlap form for r <= 2 (the C1..C4 terms of shear/src/main26.c:
//    1727-1741); the 3x3 pair tensors are built once per mobility build into
//    row lists and applied as a sparse block product (bd_real.cu);
//  * M_self: 1 - 6 alpha/sqrt(pi) + 40 alpha^3/(3 sqrt(pi)) on the diagonal;
//  * M_recip = sum over k != 0 of (phi(k)/V)(I - k k^T/k^2) cos(k.r_ij),
//    phi(k) = (1 - k^2/3)(1 + k^2/4a^2 + k^4/8a^4)(6 pi/k^2) exp(-k^2/4a^2)
//    (the coefficient of shear/src/main26.c:1622), evaluated by smooth PME
//    (Essmann et al., J. Chem. Phys. 103, 8577 (1995)) on the deforming
//    cell: fractional coordinates s = H^-1 r, cardinal B-splines of even
//    order p on a K^3 grid, three-component transforms (complex ones of two
//    right-hand sides at a time, or real ones of a single one), between them
//    multiplication by (phi/V)(I - k k^T/k^2) |b1 b2 b3|^2 with k = 2 pi H^-T m,
//    and interpolation with the same weights.
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
// (cuFFT for grid sizes it does not cover).  The spline weights, the columns'
// lists and the pair tensors are
// computed once per mobility build because its positions do not change during
// the Krylov solves.
#include <cufft.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "bd_ctx.cuh"
#include "bd_cell.cuh"
#include "bd_fft.cuh"
#include "bd_mesh.cuh"
#include "bd_real.cuh"

using namespace bd;

#define CU(call) BD_CU(call)
#define CF(call) BD_CF(call)

// Per bead: base grid index floor(u) and the p weights in each lattice
// direction (u = K s, s wrapped into [0,1)).  Positions held in the rotated
// frame are taken to the lab frame with (cr, sr) = (cos, sin) of the lattice
// angle, x = x' cr - y' sr, y = x' sr + y' cr (inverseCoords,
// extensional/src/main14.c:1525-1535); lab-frame positions pass (1, 0).  wx (FP32
// grids) gets the weights along the first direction rounded, pos the lab-frame
// position with the index in its fourth component.
__global__ void k_pme_weights(Cell cell, const double* __restrict__ rx,
                              const double* __restrict__ ry, const double* __restrict__ rz,
                              double cr, double sr, int N, int K, int p, int* base, double* w,
                              float* wx,
                              double4* pos, int* err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double x = rx[i] * cr - ry[i] * sr, y = rx[i] * sr + ry[i] * cr, z = rz[i];
  pos[i] = make_double4(x, y, z, __longlong_as_double((long long)i));
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
    double* wd = w + ((size_t)3 * i + d) * kMaxOrder;
    bspline(f, p, wd);
    if (wx && d == 0)
      for (int k = 0; k < p; k++) wx[(size_t)i * kMaxOrder + k] = (float)wd[k];
  }
}

// Right-hand sides are packed in pairs: 2p and 2p + 1 are the real and
// imaginary parts of one complex grid of three components (the component
// fastest, pair p from 3 p K^3 on).  The influence tensor is real and even in
// k, so one complex transform, the multiplication and the inverse transform
// give both products, with no unpacking.  An odd last right-hand side, or a
// single one, has a zero imaginary part.

// The influence tensor on spectra of cuFFT's, for grid sizes that bd_fft.cuh does
// not cover (thread per point and pair), the components n entries apart: a single
// right-hand side's half spectrum, or the full spectrum of packed pairs, where
// points with m2 > K/2 take the tensor of their mirror -m.
template <bool HALF, typename R, typename Cx>
__global__ void k_pme_apply_influence(const R* __restrict__ infl, Cx* spec, int K, size_t n,
                                      size_t np) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * np) return;
  const size_t m = e % n;
  size_t at = m;
  if constexpr (!HALF) {
    const int Kh = K / 2 + 1;
    int m0 = (int)(m / ((size_t)K * K)), m1 = (int)((m / K) % K), m2 = (int)(m % K);
    if (m2 > K / 2) {
      m0 = (K - m0) % K;
      m1 = (K - m1) % K;
      m2 = K - m2;
    }
    at = ((size_t)m0 * K + m1) * Kh + m2;
  }
  const R* t = infl + 6 * at;
  Cx* b = spec + 3 * n * (e / n) + m;
  Cx x = b[0], y = b[n], z = b[2 * n];
  Cx u, v, ww;
  u.x = t[0] * x.x + t[1] * y.x + t[2] * z.x;
  u.y = t[0] * x.y + t[1] * y.y + t[2] * z.y;
  v.x = t[1] * x.x + t[3] * y.x + t[4] * z.x;
  v.y = t[1] * x.y + t[3] * y.y + t[4] * z.y;
  ww.x = t[2] * x.x + t[4] * y.x + t[5] * z.x;
  ww.y = t[2] * x.y + t[4] * y.y + t[5] * z.y;
  b[0] = u;
  b[n] = v;
  b[2 * n] = ww;
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

namespace bd {

// cuFFT plan of `batch` contiguous grids, distances id and od apart.
static int make_plan(bd_ctx* c, int* slot, int id, int od, cufftType type, int batch) {
  int n[3] = {c->pmeK, c->pmeK, c->pmeK};
  cufftHandle f;
  CF(cufftPlanMany(&f, 3, n, nullptr, 1, id, nullptr, 1, od, type, batch));
  *slot = (int)f + 1;
  CF(cufftSetStream(f, c->stream));
  return BD_OK;
}

static void drop_plan(int* plan) {
  if (*plan) cufftDestroy((cufftHandle)(*plan - 1));
  *plan = 0;
}

// In-place transforms of the packed pairs of k right-hand sides, for grid sizes
// bd_fft.cuh does not cover: one plan for all their grids, made outside any
// capture and kept for up to four numbers of pairs (replacing one drops the
// captured iterations that use it).
int pme_pairs_plan(bd_ctx* c, int k) {
  if (!c->pme_planar || k < 2) return BD_OK;
  const int np = (k + 1) / 2;
  int slot = -1;
  for (int q = 3; q >= 0; q--) {
    if (c->pme_mplan[q] && c->pme_mplan_np[q] == np) return BD_OK;
    if (!c->pme_mplan[q]) slot = q;
  }
  if (slot < 0) {
    slot = 3;
    lanczos_graphs_reset(c);
    drop_plan(&c->pme_mplan[slot]);
  }
  const int K3 = c->pmeK * c->pmeK * c->pmeK;
  c->pme_mplan_np[slot] = np;
  const int s = make_plan(c, &c->pme_mplan[slot], K3, K3, c->pme_f32 ? CUFFT_C2C : CUFFT_Z2Z, 3 * np);
  if (s != BD_OK) drop_plan(&c->pme_mplan[slot]);
  return s;
}

// Whether a single right-hand side on a grid that bd_fft.cuh covers goes through
// cuFFT's real transforms: half the data, but a pass more and planar grids.
// Products by them and by the five complex passes, us, FP64: 80^3 140 and 130, 96^3
// 214 and 193, 100^3 179 and 212, 128^3 324 and 452, 135^3 514 and 495, 144^3 425
// and 591, 225^3 2052 and 2384, 256^3 2263 and 3532.  FP32: 120^3 218 and 206, 128^3
// 235 and 236 (a thousand beads 127 and 149), 144^3 302 and 321, 150^3 425 and 381,
// 160^3 444 and 468, 192^3 698 and 781, 240^3 1550 and 1486, 256^3 1502 and 1730.
static bool real_single(int K, bool f32) {
  return f32 ? K >= 128 && K % 16 == 0 && K % 15 != 0 : K >= 100 && (K % 2 == 0 || K > 200);
}

static int pme_parts(bd_ctx* c) {
  int s, K = c->pmeK, N = c->N;
  size_t K3 = (size_t)K * K * K, Ks = (size_t)K * K * (K / 2 + 1);
  c->pme_f32 = c->p.precision == BD_PREC_FP32;
  size_t es = c->pme_f32 ? 4 : 8;  // grid, spectrum, influence and pair tensors
  c->pme_planar = !fft_has_size(K);
  c->pme_real1 = c->pme_planar || real_single(K, c->pme_f32);
  // the packed pairs' grids for the largest number of right-hand sides; with
  // pme_real1 a single one's real grids and behind them its half spectra
  size_t nr = (size_t)std::max(1, c->nbk);
  size_t real_bytes = (es * 3 * K3 + 255) / 256 * 256;
  size_t grid_bytes = c->pme_real1 && nr == 1 ? 0 : 2 * es * 3 * K3 * ((nr + 1) / 2);
  if (c->pme_real1) grid_bytes = std::max(grid_bytes, real_bytes + 2 * es * 3 * Ks);
  c->pme_nblk = (int)((Ks + 255) / 256);
  s = alloc_all(c, {{&c->pme_grid, grid_bytes},
                    {&c->pme_tw, 2 * es * K},
                    {&c->pme_infl, es * 6 * Ks},
                    {&c->pme_bsq, 8 * 3 * (size_t)K},
                    {&c->pme_soff, 8 * (3 * (size_t)c->pme_nblk + 3)},
                    {&c->pme_base, 4 * 3 * (size_t)N},
                    {&c->pme_w, 8 * 3 * (size_t)N * kMaxOrder},
                    {&c->pme_vpk, 6 * es * (size_t)N * ((nr + 1) / 2)},
                    {&c->rl_pos, 32 * (size_t)N}});
  if (s == BD_OK && c->pme_f32) s = alloc_all(c, {{&c->pme_wx, 4 * (size_t)N * kMaxOrder}});
  if (s != BD_OK || (s = mesh_alloc(c)) != BD_OK || (s = real_alloc(c)) != BD_OK) return s;
  if (c->pme_real1) {
    c->pme_spec = (char*)c->pme_grid + real_bytes;
    const bool f32 = c->pme_f32;
    const int nk = (int)K3, nh = (int)Ks;
    if ((s = make_plan(c, &c->pme_plan_f, nk, nh, f32 ? CUFFT_R2C : CUFFT_D2Z, 3)) != BD_OK ||
        (s = make_plan(c, &c->pme_plan_b, nh, nk, f32 ? CUFFT_C2R : CUFFT_Z2D, 3)) != BD_OK)
      return s;
  }
  if (c->pme_planar && nr > 1 && (s = pme_pairs_plan(c, (int)nr)) != BD_OK) return s;
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
  for (int* plan : {&c->pme_plan_f, &c->pme_plan_b, &c->pme_mplan[0], &c->pme_mplan[1],
                    &c->pme_mplan[2], &c->pme_mplan[3]})
    drop_plan(plan);
  mesh_free(c);
  real_free(c);
  free_all({&c->pme_vpk, &c->pme_grid, &c->pme_tw, &c->pme_infl, &c->pme_bsq, &c->pme_soff,
            &c->pme_base, &c->pme_w, &c->pme_wx, &c->rl_pos});
}

// The mobility's buffers and plan, all or none (pme_grid tells).
static int pme_alloc(bd_ctx* c) {
  if (c->pme_grid) return BD_OK;
  const size_t before = c->bytes;
  const int s = pme_parts(c);
  if (s != BD_OK) {
    pme_free(c);
    c->bytes = before;
  }
  return s;
}

// Preparation for the current positions, in the frame calcHI reads them
// (extension: rotated by the lattice angle, taken to the lab frame here):
// spline weights, influence tensor of the current cell, self off-diagonal
// sums, real-space pair list and tensors.  The products that follow use this
// configuration until the next preparation, as the dense matrix does.
int pme_prepare(bd_ctx* c, const Lat& l) {
  int s;
  c->pme_ready = c->hi_built = false;  // until it is complete
  if ((s = pme_alloc(c)) != BD_OK || (s = real_rows(c)) != BD_OK) return s;
  Cell cell = make_cell(l);
  double cr = 1.0, sr = 0.0;
  if (l.flow == BD_FLOW_EXT) {
    cr = l.cth;
    sr = l.sth;
  }
  double alpha = c->pme_alpha;
  int K = c->pmeK, N = c->N;
  // calcHI's split parameter at this step, for its overlap convention
  double rce = l.treal <= c->tp / 2 ? l.L2yp : 2.0 * l.L2yp;
  double alpha_ref = 4.0 / rce;
  c->launches += 3;
  k_pme_weights<<<nblk(N, 128), 128, 0, c->stream>>>(cell, c->rx, c->ry, c->rz, cr, sr, N, K,
                                                     c->pme_p, c->pme_base, c->pme_w, c->pme_wx,
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
  if ((s = real_prepare(c, l, cell, cr, sr, alpha_ref)) != BD_OK) return s;
  double a = alpha;
  c->pme_self = 1.0 - 6.0 / sqrt(M_PI) * a + 40.0 / (3.0 * sqrt(M_PI)) * a * a * a;
  c->Dtr[0] = c->Dtr[1] = c->Dtr[2] = c->pme_self;
  c->pme_ready = true;
  c->hi_built = true;
  return launch_ok(c);
}

// The transforms through cuFFT, for grid sizes bd_fft.cuh does not cover: single
// right-hand sides by real transforms, packed pairs all at once in place.
// The grids hold their components one after the other: interleaved ones (element
// stride 3) cost cuFFT more than the transforms themselves.  30 000 beads on 125^3,
// ten vectors FP32, one FP32, one FP64: 1263, 226, 304 us; interleaved, a pair at a
// time and complex throughout 1767, 376, 603.  150 000 on 216^3: 5637, 951, 1377;
// 10400, 2100, 4080.
template <typename R, typename Cx>
static int cufft_influence(bd_ctx* c, int k) {
  const int K = c->pmeK, np = (k + 1) / 2;
  const size_t K3 = (size_t)K * K * K, Ks = (size_t)K * K * (K / 2 + 1);
  constexpr bool F = sizeof(R) == 4;
  c->launches++;
  if (k == 1) {
    const cufftHandle f = (cufftHandle)(c->pme_plan_f - 1), b = (cufftHandle)(c->pme_plan_b - 1);
    if constexpr (F)
      CF(cufftExecR2C(f, (cufftReal*)c->pme_grid, (cufftComplex*)c->pme_spec));
    else
      CF(cufftExecD2Z(f, (cufftDoubleReal*)c->pme_grid, (cufftDoubleComplex*)c->pme_spec));
    k_pme_apply_influence<true, R, Cx><<<nblk((long long)Ks, 256), 256, 0, c->stream>>>(
        (const R*)c->pme_infl, (Cx*)c->pme_spec, K, Ks, 1);
    if constexpr (F)
      CF(cufftExecC2R(b, (cufftComplex*)c->pme_spec, (cufftReal*)c->pme_grid));
    else
      CF(cufftExecZ2D(b, (cufftDoubleComplex*)c->pme_spec, (cufftDoubleReal*)c->pme_grid));
    return BD_OK;
  }
  int q = 0;
  while (q < 4 && !(c->pme_mplan[q] && c->pme_mplan_np[q] == np)) q++;
  if (q == 4) return BD_ERR_STATE;  // pme_pairs_plan(c, k) first
  for (int dir : {CUFFT_FORWARD, CUFFT_INVERSE}) {
    const cufftHandle f = (cufftHandle)(c->pme_mplan[q] - 1);
    Cx* g = (Cx*)c->pme_grid;
    if constexpr (F)
      CF(cufftExecC2C(f, (cufftComplex*)g, (cufftComplex*)g, dir));
    else
      CF(cufftExecZ2Z(f, (cufftDoubleComplex*)g, (cufftDoubleComplex*)g, dir));
    if (dir == CUFFT_FORWARD)
      k_pme_apply_influence<false, R, Cx><<<nblk((long long)K3 * np, 256), 256, 0, c->stream>>>(
          (const R*)c->pme_infl, g, K, K3, (size_t)np);
  }
  return BD_OK;
}

// out_r = M v_r by PME for k right-hand sides given by component pointers
// (VecIn) and RHS strides vr (input) and orr (output).
template <typename R, typename Cx>
static int pme_apply_t(bd_ctx* c, int k, const VecIn& v, size_t vr, double* o0, double* o1,
                       double* o2, int ostride, size_t orr) {
  int K = c->pmeK, N = c->N, s;
  if (k < 1 || k > std::max(1, c->nbk)) return BD_ERR_ARG;
  int np = (k + 1) / 2;
  Cx* g = (Cx*)c->pme_grid;
  if ((s = mesh_spread(c, k, v, vr, g)) != BD_OK) return s;
  if (k == 1 ? c->pme_real1 : c->pme_planar)
    s = cufft_influence<R, Cx>(c, k);
  else
    s = sizeof(R) == 4 ? fft_influence_f32(c, K, g, np, c->pme_infl, c->pme_tw)
                       : fft_influence_f64(c, K, g, np, c->pme_infl, c->pme_tw);
  if (s != BD_OK) return s;
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
  return real_apply(c, np, fin);
}

// Forward transform, tensor and inverse transform of one packed pair's grid, as a
// product runs them.
static int transform_pair(bd_ctx* c) {
  if (c->pme_planar)
    return c->pme_f32 ? cufft_influence<float, cufftComplex>(c, 2)
                      : cufft_influence<double, cufftDoubleComplex>(c, 2);
  return (c->pme_f32 ? fft_influence_f32 : fft_influence_f64)(c, c->pmeK, c->pme_grid, 1,
                                                              c->pme_infl, c->pme_tw);
}

// Time of one packed pair's transforms on K^3 points, on the default stream.
int pme_time_transforms(int K, bool f32, float* ms) {
  bd_ctx* c = new bd_ctx();  // a workspace without beads
  c->pmeK = K;
  c->pme_p = 8;
  c->p.precision = f32 ? BD_PREC_FP32 : BD_PREC_FP64;
  c->nbk = 2;
  c->boxvol = 1.0;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto run = [&]() -> int {
    int s = pme_alloc(c);
    if (s != BD_OK) return s;
    const size_t es = f32 ? 4 : 8, K3 = (size_t)K * K * K, Ks = (size_t)K * K * (K / 2 + 1);
    CU(cudaMemsetAsync(c->pme_grid, 0, 6 * es * K3, c->stream));
    CU(cudaMemsetAsync(c->pme_infl, 0, 6 * es * Ks, c->stream));
    CU(cudaEventCreate(&e0));
    CU(cudaEventCreate(&e1));
    for (int rep = 0; rep < 8; rep++) {
      if (rep == 3) CU(cudaEventRecord(e0, c->stream));
      if ((s = transform_pair(c)) != BD_OK) return s;
    }
    CU(cudaEventRecord(e1, c->stream));
    CU(cudaEventSynchronize(e1));
    CU(cudaEventElapsedTime(ms, e0, e1));
    *ms /= 5;
    return launch_ok(c);
  };
  const int s = run();
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  pme_free(c);
  delete c;
  return s;
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
