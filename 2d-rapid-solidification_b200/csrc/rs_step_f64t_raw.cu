// rs_step_f64t_raw.cu — the FP64 tile kernels of fields whose rows are not
// 16-byte aligned (rs_tile_f64.cuh).
#include "rs_tile_f64.cuh"

namespace rs {

StepKernel64 raw_kernel_f64(int rows, bool own) {
  if (rows == 4) return {own ? tile_kernel_f64<4, false, true, true> : tile_kernel_f64<4, false, true>, sizeof(TileOps<4>::TileSmem<false>)};
  if (rows == 8) return {tile_kernel_f64<8, false, true>, sizeof(TileOps<8>::TileSmem<false>)};
  return {tile_kernel_f64<16, false, true>, sizeof(TileOps<16>::TileSmem<false>)};
}

}  // namespace rs
