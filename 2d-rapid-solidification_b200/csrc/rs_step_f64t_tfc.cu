// rs_step_f64t_tfc.cu — the FP64 tile kernels of the coarse-grid temperature
// (rs_tile_f64.cuh).
#include "rs_tile_f64.cuh"

namespace rs {

StepKernel64 tfc_kernel_f64(int rows) {
  if (rows == 8) return {tile_kernel_f64<8, true, false>, sizeof(TileOps<8>::TileSmem<true>)};
  return {tile_kernel_f64<16, true, false>, sizeof(TileOps<16>::TileSmem<true>)};
}

}  // namespace rs
