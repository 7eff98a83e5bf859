// rs_step_f32_tfc.cu — the FP32 tile kernels of the coarse-grid temperature
// (rs_tile_f32.cuh).
#include "rs_tile_f32.cuh"

namespace rs {

ExactKernel32 tfc_kernel_f32(bool raw) {
  return {raw ? tile_kernel_tfc<true> : tile_kernel_tfc<false>, sizeof(TileSmemT<kTfcTR, true>)};
}

}  // namespace rs
