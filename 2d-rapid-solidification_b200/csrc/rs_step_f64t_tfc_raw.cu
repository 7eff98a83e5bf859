// rs_step_f64t_tfc_raw.cu — the FP64 tile kernels of the coarse-grid temperature,
// fields whose rows are not 16-byte aligned (rs_tile_f64.cuh).
#include "rs_tile_f64.cuh"

namespace rs {

StepKernel64 tfc_raw_kernel_f64(int rows) {
  if (rows == 8) return {tile_kernel_f64<8, true, true>, sizeof(TileOps<8>::TileSmem<true>)};
  return {tile_kernel_f64<16, true, true>, sizeof(TileOps<16>::TileSmem<true>)};
}

}  // namespace rs
