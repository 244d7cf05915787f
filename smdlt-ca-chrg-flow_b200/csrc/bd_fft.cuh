// Three-dimensional complex transforms of the packed-pair grids, with the
// mobility's influence tensor applied between them.
//
// No counterpart in the reference (see bd_pme.cu).  A grid holds, per packed
// pair of right-hand sides, K^3 points of three complex components, the
// component fastest: the product's spreading and interpolation touch a point's
// components together, and the influence tensor mixes them.  cuFFT transforms
// such a grid only with strided batches (and a pass of its own for the
// tensor); these kernels do
//   z forward, y forward, x forward + tensor + x inverse, y inverse, z inverse
// in five passes over the grid instead of seven.
//
// A line of K = R1 R2 points is transformed in two steps (Cooley and Tukey,
// Math. Comp. 19, 297 (1965)): a thread loads the R1 points n2 + R2 n1 of its
// column straight from memory, transforms them in registers, multiplies by the
// twiddles exp(-2 pi i n2 k1 / K) and passes them on through shared memory; a
// thread then takes the R2 values of its k1, transforms them and stores the
// points k1 + R1 k2.  Every point is read and written once per pass, 24 or 48
// contiguous bytes and more at a time.  The inverse is the same kernel with
// real and imaginary parts exchanged at both ends.
// Bound by the grid's round trip through L2 and HBM.  Five pairs, forward,
// tensor and inverse: 251 us on 100^3 FP32 (cuFFT's six passes and the tensor's
// 330), 63 us on 64^3 FP32 (88), 107 us on 64^3 FP64 (148).
#pragma once

#include <type_traits>
#include <utility>

#include "bd_ctx.cuh"

namespace fft {

template <typename R>
struct Cplx;
template <>
struct Cplx<float> {
  using T = float2;
};
template <>
struct Cplx<double> {
  using T = double2;
};

// cos and sin of 2 pi m / n at compile time: Taylor series on [-pi, pi].
constexpr double kPi = 3.14159265358979323846;
__host__ __device__ constexpr double turn(int m, int n) {
  m %= n;
  if (2 * m > n) m -= n;
  return 2.0 * kPi * m / n;
}
__host__ __device__ constexpr double taylor(double x, double term, int k0) {
  double s = term;
  for (int k = k0; k < k0 + 40; k += 2) {
    term *= -x * x / (double)(k * (k + 1));
    s += term;
  }
  return s;
}
// on quarter turns and below, so that no large terms cancel
__host__ __device__ constexpr double ccos(int m, int n);
__host__ __device__ constexpr double csin(int m, int n) {
  double x = turn(m, n);
  if (x > kPi / 2) return taylor(kPi - x, kPi - x, 2);
  if (x < -kPi / 2) return -taylor(kPi + x, kPi + x, 2);
  return taylor(x, x, 2);
}
__host__ __device__ constexpr double ccos(int m, int n) {
  double x = turn(m, n);
  if (x < 0) x = -x;
  if (x > kPi / 2) return -taylor(kPi - x, 1.0, 1);
  return taylor(x, 1.0, 1);
}

template <class F, int... I>
__device__ __forceinline__ void static_for_(F f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>()), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F f) {
  static_for_(f, std::make_integer_sequence<int, N>());
}

template <class C>
__device__ __forceinline__ C add(C a, C b) {
  a.x += b.x;
  a.y += b.y;
  return a;
}
template <class C>
__device__ __forceinline__ C sub(C a, C b) {
  a.x -= b.x;
  a.y -= b.y;
  return a;
}
template <class C>
__device__ __forceinline__ C mul(C a, C w) {
  C r;
  r.x = a.x * w.x - a.y * w.y;
  r.y = a.x * w.y + a.y * w.x;
  return r;
}
template <class C>
__device__ __forceinline__ C swapped(C a, bool on) {
  C r;
  r.x = on ? a.y : a.x;
  r.y = on ? a.x : a.y;
  return r;
}

// Forward transform of R values in registers, X[k] = sum_n x[n] exp(-2 pi i n k/R).
template <int R>
struct Split {  // R = A B
  static constexpr int A = R % 4 == 0 && R != 8 && R != 12 ? 4 : R % 2 == 0 && R != 12 ? 2 : 3;
  static constexpr int B = R / A;
};

template <int R, class C>
__device__ __forceinline__ void dft(C (&x)[R]) {
  using T = decltype(x[0].x);
  using V = std::remove_reference_t<T>;
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    C a = x[0];
    x[0] = add(a, x[1]);
    x[1] = sub(a, x[1]);
  } else if constexpr (R == 3) {
    constexpr V s = (V)0.86602540378443864676;
    C t = add(x[1], x[2]), d = sub(x[1], x[2]), m = x[0];
    m.x -= (V)0.5 * t.x;
    m.y -= (V)0.5 * t.y;
    x[0] = add(x[0], t);
    x[1].x = m.x + s * d.y;
    x[1].y = m.y - s * d.x;
    x[2].x = m.x - s * d.y;
    x[2].y = m.y + s * d.x;
  } else if constexpr (R == 4) {
    C a = add(x[0], x[2]), b = sub(x[0], x[2]), c = add(x[1], x[3]), d = sub(x[1], x[3]);
    x[0] = add(a, c);
    x[2] = sub(a, c);
    x[1].x = b.x + d.y;
    x[1].y = b.y - d.x;
    x[3].x = b.x - d.y;
    x[3].y = b.y + d.x;
  } else if constexpr (R == 5) {
    constexpr V c1 = (V)ccos(1, 5), c2 = (V)ccos(2, 5), s1 = (V)csin(1, 5), s2 = (V)csin(2, 5);
    C p = add(x[1], x[4]), q = add(x[2], x[3]), u = sub(x[1], x[4]), v = sub(x[2], x[3]);
    C a, b, m, n;
    a.x = x[0].x + c1 * p.x + c2 * q.x;
    a.y = x[0].y + c1 * p.y + c2 * q.y;
    b.x = x[0].x + c2 * p.x + c1 * q.x;
    b.y = x[0].y + c2 * p.y + c1 * q.y;
    m.x = s1 * u.x + s2 * v.x;
    m.y = s1 * u.y + s2 * v.y;
    n.x = s2 * u.x - s1 * v.x;
    n.y = s2 * u.y - s1 * v.y;
    x[0] = add(x[0], add(p, q));
    x[1].x = a.x + m.y;
    x[1].y = a.y - m.x;
    x[4].x = a.x - m.y;
    x[4].y = a.y + m.x;
    x[2].x = b.x + n.y;
    x[2].y = b.y - n.x;
    x[3].x = b.x - n.y;
    x[3].y = b.y + n.x;
  } else {
    constexpr int A = Split<R>::A, B = Split<R>::B;
    C y[R];  // y[B k1 + b]
    static_for<B>([&](auto bI) {
      constexpr int b = decltype(bI)::value;
      C t[A];
#pragma unroll
      for (int a = 0; a < A; a++) t[a] = x[B * a + b];
      dft<A>(t);
      static_for<A>([&](auto kI) {
        constexpr int k = decltype(kI)::value;
        if constexpr (b * k == 0) {
          y[B * k + b] = t[k];
        } else {
          constexpr V wr = (V)ccos(b * k, R), wi = (V)-csin(b * k, R);
          C w;
          w.x = wr;
          w.y = wi;
          y[B * k + b] = mul(t[k], w);
        }
      });
    });
#pragma unroll
    for (int k = 0; k < A; k++) {
      C t[B];
#pragma unroll
      for (int b = 0; b < B; b++) t[b] = y[B * k + b];
      dft<B>(t);
#pragma unroll
      for (int q = 0; q < B; q++) x[k + A * q] = t[q];
    }
  }
}

// Lines along z: K points of three components, contiguous.  A block takes NL
// lines; step one by a thread per (line, n2, component), step two per (line,
// k1, component).  The rows of the exchange are padded so that consecutive
// (k1, component) start three elements apart modulo the banks.
template <int R1, int R2, typename R>
__global__ void __launch_bounds__(384) k_fft_z(typename Cplx<R>::T* g, size_t nlines, int NL,
                                               const typename Cplx<R>::T* __restrict__ tw,
                                               int inv) {
  using C = typename Cplx<R>::T;
  constexpr int K = R1 * R2, M = sizeof(R) == 4 ? 16 : 8;
  constexpr int ROW = 3 * R2 + ((3 - 3 * R2) % M + M) % M, LS = R1 * ROW;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* s = (C*)fft_smem;
  const size_t l0 = (size_t)blockIdx.x * NL;
  const int nl = (int)min((size_t)NL, nlines - l0);
  C* p = g + l0 * 3 * K;
  for (int t = threadIdx.x; t < nl * 3 * R2; t += blockDim.x) {
    const int line = t / (3 * R2), nc = t % (3 * R2), n2 = nc / 3;
    C x[R1];
#pragma unroll
    for (int a = 0; a < R1; a++) x[a] = swapped(p[(size_t)line * 3 * K + 3 * R2 * a + nc], inv);
    dft<R1>(x);
#pragma unroll
    for (int a = 0; a < R1; a++)
      s[line * LS + a * ROW + nc] = a == 0 ? x[a] : mul(x[a], __ldg(tw + n2 * a));
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nl * 3 * R1; t += blockDim.x) {
    const int line = t / (3 * R1), kc = t % (3 * R1), k1 = kc / 3, c = kc % 3;
    C x[R2];
#pragma unroll
    for (int b = 0; b < R2; b++) x[b] = s[line * LS + k1 * ROW + 3 * b + c];
    dft<R2>(x);
#pragma unroll
    for (int b = 0; b < R2; b++) p[(size_t)line * 3 * K + 3 * R1 * b + kc] = swapped(x[b], inv);
  }
}

// Lines of stride `inner` (y: 3 K): columns (outer, i), i < inner fastest; a
// block takes TI consecutive columns.
template <int R1, int R2, typename R, int TI>
__global__ void __launch_bounds__(TI * (R1 > R2 ? R1 : R2))
    k_fft_y(typename Cplx<R>::T* g, size_t ncol, int inner,
            const typename Cplx<R>::T* __restrict__ tw, int inv) {
  using C = typename Cplx<R>::T;
  constexpr int K = R1 * R2;
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* s = (C*)fft_smem;
  const int col = threadIdx.x % TI, row = threadIdx.x / TI;
  const size_t q = (size_t)blockIdx.x * TI + col;
  const bool in = q < ncol;
  C* p = g + (q / inner) * (size_t)K * inner + q % inner;
  if (in && row < R2) {
    C x[R1];
#pragma unroll
    for (int a = 0; a < R1; a++) x[a] = swapped(p[(size_t)(row + R2 * a) * inner], inv);
    dft<R1>(x);
#pragma unroll
    for (int a = 0; a < R1; a++)
      s[(a * R2 + row) * TI + col] = a == 0 ? x[a] : mul(x[a], __ldg(tw + row * a));
  }
  __syncthreads();
  if (in && row < R1) {
    C x[R2];
#pragma unroll
    for (int b = 0; b < R2; b++) x[b] = s[(row * R2 + b) * TI + col];
    dft<R2>(x);
#pragma unroll
    for (int b = 0; b < R2; b++) p[(size_t)(row + R1 * b) * inner] = swapped(x[b], inv);
  }
}

// Lines along x, forward, times the influence tensor, inverse: TI (a multiple
// of 3) consecutive columns (y, z, component) of one pair.  The spectrum
// stays in shared memory, index k1 + R1 k2 at row k1 R2 + k2: the second
// forward step and the first inverse step each work on a thread's own row.
// The tensor (six real numbers per point of the half spectrum, even in k):
// points with m2 > K/2 take that of their mirror -m.
template <int R1, int R2, typename R, int TI>
__global__ void __launch_bounds__(TI * (R1 > R2 ? R1 : R2))
    k_fft_x(typename Cplx<R>::T* g, const R* __restrict__ infl,
            const typename Cplx<R>::T* __restrict__ tw) {
  using C = typename Cplx<R>::T;
  constexpr int K = R1 * R2, Kh = K / 2 + 1, inner = 3 * K * K;
  static_assert(TI % 3 == 0, "a point's components stay together");
  extern __shared__ __align__(16) unsigned char fft_smem[];
  C* s = (C*)fft_smem;
  const int col = threadIdx.x % TI, row = threadIdx.x / TI;
  const int i0 = blockIdx.x * TI;
  const bool in = i0 + col < inner;
  C* p = g + (size_t)blockIdx.y * K * inner + i0 + col;
  if (in && row < R2) {
    C x[R1];
#pragma unroll
    for (int a = 0; a < R1; a++) x[a] = p[(size_t)(row + R2 * a) * inner];
    dft<R1>(x);
#pragma unroll
    for (int a = 0; a < R1; a++)
      s[(a * R2 + row) * TI + col] = a == 0 ? x[a] : mul(x[a], __ldg(tw + row * a));
  }
  __syncthreads();
  if (in && row < R1) {
    C x[R2];
#pragma unroll
    for (int b = 0; b < R2; b++) x[b] = s[(row * R2 + b) * TI + col];
    dft<R2>(x);
#pragma unroll
    for (int b = 0; b < R2; b++) s[(row * R2 + b) * TI + col] = x[b];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < K * (TI / 3); t += blockDim.x) {
    const int j = t % (TI / 3), r = t / (TI / 3), i = i0 / 3 + j;
    if (i >= K * K) continue;
    int m0 = r / R2 + R1 * (r % R2), m1 = i / K, m2 = i % K;
    if (m2 > K / 2) {
      m0 = m0 ? K - m0 : 0;
      m1 = m1 ? K - m1 : 0;
      m2 = K - m2;
    }
    const C* w = (const C*)infl + 3 * (((size_t)m0 * K + m1) * Kh + m2);
    const C wa = __ldg(w), wb = __ldg(w + 1), wc = __ldg(w + 2);  // xx xy, xz yy, yz zz
    C* q = s + r * TI + 3 * j;
    C x = q[0], y = q[1], z = q[2], u, v, ww;
    u.x = wa.x * x.x + wa.y * y.x + wb.x * z.x;
    u.y = wa.x * x.y + wa.y * y.y + wb.x * z.y;
    v.x = wa.y * x.x + wb.y * y.x + wc.x * z.x;
    v.y = wa.y * x.y + wb.y * y.y + wc.x * z.y;
    ww.x = wb.x * x.x + wc.x * y.x + wc.y * z.x;
    ww.y = wb.x * x.y + wc.x * y.y + wc.y * z.y;
    q[0] = swapped(u, true);  // the inverse below is the forward transform swapped
    q[1] = swapped(v, true);
    q[2] = swapped(ww, true);
  }
  __syncthreads();
  if (in && row < R1) {
    C x[R2];
#pragma unroll
    for (int b = 0; b < R2; b++) x[b] = s[(row * R2 + b) * TI + col];
    dft<R2>(x);
#pragma unroll
    for (int b = 0; b < R2; b++)
      s[(row * R2 + b) * TI + col] = b == 0 ? x[b] : mul(x[b], __ldg(tw + row * b));
  }
  __syncthreads();
  if (in && row < R2) {
    C x[R1];
#pragma unroll
    for (int a = 0; a < R1; a++) x[a] = s[(a * R2 + row) * TI + col];
    dft<R1>(x);
#pragma unroll
    for (int a = 0; a < R1; a++) p[(size_t)(row + R2 * a) * inner] = swapped(x[a], true);
  }
}

// The five passes for one size.
template <int R1, int R2, typename R>
int run(bd_ctx* c, void* grid, int np, const void* infl, const void* tw) {
  using C = typename Cplx<R>::T;
  constexpr int K = R1 * R2, RM = R1 > R2 ? R1 : R2, TY = sizeof(R) == 4 ? 32 : 16, TX = 24;
  constexpr int M = sizeof(R) == 4 ? 16 : 8;
  constexpr int ROW = 3 * R2 + ((3 - 3 * R2) % M + M) % M;
  C* g = (C*)grid;
  const C* w = (const C*)tw;
  const size_t lines = (size_t)np * K * K;
  // as many z lines as give a block about 320 threads
  constexpr int NL = 3 * RM >= 320 ? 1 : 320 / (3 * RM), TZ = (NL * 3 * RM + 31) / 32 * 32;
  constexpr size_t sz = sizeof(C) * (size_t)NL * R1 * ROW, sy = sizeof(C) * (size_t)K * TY,
                   sx = sizeof(C) * (size_t)K * TX;
  static_assert(TZ <= 384, "block size of the z pass");
  if constexpr (sz > 48 * 1024)
    BD_CU(cudaFuncSetAttribute(k_fft_z<R1, R2, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sz));
  if constexpr (sy > 48 * 1024)
    BD_CU(cudaFuncSetAttribute(k_fft_y<R1, R2, R, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy));
  if constexpr (sx > 48 * 1024)
    BD_CU(cudaFuncSetAttribute(k_fft_x<R1, R2, R, TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
  const unsigned bz = (unsigned)((lines + NL - 1) / NL);
  const size_t ncol = (size_t)np * K * 3 * K;
  const unsigned by = (unsigned)((ncol + TY - 1) / TY);
  const dim3 bx((3 * K * K + TX - 1) / TX, np);
  c->launches += 5;
  k_fft_z<R1, R2, R><<<bz, TZ, sz, c->stream>>>(g, lines, NL, w, 0);
  k_fft_y<R1, R2, R, TY><<<by, TY * RM, sy, c->stream>>>(g, ncol, 3 * K, w, 0);
  k_fft_x<R1, R2, R, TX><<<bx, TX * RM, sx, c->stream>>>(g, (const R*)infl, w);
  k_fft_y<R1, R2, R, TY><<<by, TY * RM, sy, c->stream>>>(g, ncol, 3 * K, w, 1);
  k_fft_z<R1, R2, R><<<bz, TZ, sz, c->stream>>>(g, lines, NL, w, 1);
  return BD_OK;
}

// The sizes with a pair of factors up to 16 that the transforms in registers
// cover: every 2^a 3^b 5^c from 20 to 160 but 125, and up to 256 those that are
// not 162, 200, 216, 243 or 250.  Other sizes go through cuFFT (bd_pme.cu).
#define BD_FFT_SIZES(X)                                                                       \
  X(4, 5) X(4, 6) X(5, 5) X(3, 9) X(5, 6) X(4, 8) X(6, 6) X(5, 8) X(5, 9) X(6, 8) X(5, 10)    \
  X(6, 9) X(6, 10) X(8, 8) X(8, 9) X(5, 15) X(8, 10) X(9, 9) X(9, 10) X(8, 12) X(10, 10)      \
  X(9, 12) X(10, 12) X(8, 16) X(9, 15) X(12, 12) X(10, 15) X(10, 16) X(12, 15) X(12, 16)      \
  X(15, 15) X(15, 16) X(16, 16)

inline bool has_size(int K) {
#define BD_FFT_CASE(A, B) \
  if (K == (A) * (B)) return true;
  BD_FFT_SIZES(BD_FFT_CASE)
#undef BD_FFT_CASE
  return false;
}

template <typename R>
int run_size(bd_ctx* c, int K, void* grid, int np, const void* infl, const void* tw) {
  switch (K) {
#define BD_FFT_CASE(A, B) \
  case (A) * (B):         \
    return run<A, B, R>(c, grid, np, infl, tw);
    BD_FFT_SIZES(BD_FFT_CASE)
#undef BD_FFT_CASE
  }
  return BD_ERR_STATE;
}

}  // namespace fft

namespace bd {
// Forward transform, influence tensor, inverse transform of np packed-pair
// grids of K^3 points in place; tw holds exp(-2 pi i m / K), m < K.
int fft_influence_f32(bd_ctx* c, int K, void* grid, int np, const void* infl, const void* tw);
int fft_influence_f64(bd_ctx* c, int K, void* grid, int np, const void* infl, const void* tw);
bool fft_has_size(int K);
}  // namespace bd
