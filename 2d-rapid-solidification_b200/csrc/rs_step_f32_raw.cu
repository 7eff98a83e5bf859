// rs_step_f32_raw.cu — the FP32 tile kernels of fields whose rows are not 16-byte aligned
// (rs_tile_f32.cuh).
#include "rs_tile_f32.cuh"

namespace rs {

StepKernel32 raw_kernel_f32(int rows) {
  if (rows == 4) return {tile_kernel<false, 4, true>, sizeof(TileSmemT<4>)};
  if (rows == 8) return {tile_kernel<false, 8, true>, sizeof(TileSmemT<8>)};
  return {tile_kernel<false, 16, true>, sizeof(TileSmemT<16>)};
}

}  // namespace rs
