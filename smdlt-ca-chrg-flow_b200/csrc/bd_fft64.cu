// FP64 transforms of the packed-pair grids (bd_fft.cuh).
#include "bd_fft.cuh"

namespace bd {

int fft_influence_f64(bd_ctx* c, int K, void* grid, int np, const void* infl, const void* tw) {
  return fft::run_size<double>(c, K, grid, np, infl, tw);
}

}  // namespace bd
