// Real-space part of the particle-mesh mobility (bd_real.cu) and the assembly of
// a product.
#pragma once

#include "bd_ctx.cuh"
#include "bd_cell.cuh"

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

namespace bd {
int real_alloc(bd_ctx* c);
void real_free(bd_ctx* c);
int real_rows(bd_ctx* c);
int real_prepare(bd_ctx* c, const Lat& l, const Cell& cell, double cr, double sr, double alpha_ref);
int real_apply(bd_ctx* c, int np, const Finish& fin);
}  // namespace bd
