// rs_step_f32_net.cu — the FP32 tile kernels that evaluate cells through the learned network
// (rs_tile_f32.cuh).
#include "rs_tile_f32.cuh"

namespace rs {

StepKernel32 net_kernel_f32(int rows) {
  if (rows == 4) return {tile_kernel<true, 4, false>, sizeof(TileSmemT<4>)};
  if (rows == 8) return {tile_kernel<true, 8, false>, sizeof(TileSmemT<8>)};
  return {tile_kernel<true, 16, false>, sizeof(TileSmemT<16>)};
}

}  // namespace rs
