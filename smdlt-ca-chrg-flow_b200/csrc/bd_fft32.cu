// FP32 transforms of the packed-pair grids (bd_fft.cuh).
#include "bd_fft.cuh"

namespace bd {

bool fft_has_size(int K) { return fft::has_size(K); }

int fft_influence_f32(bd_ctx* c, int K, void* grid, int np, const void* infl, const void* tw) {
  return fft::run_size<float>(c, K, grid, np, infl, tw);
}

}  // namespace bd
