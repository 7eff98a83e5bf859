// rs_step_f64t_raw.cu — the FP64 tile kernels of fields whose rows are not
// 16-byte aligned (rs_tile_f64.cuh).
#include "rs_tile_f64.cuh"

namespace rs {

StepKernel64 raw_kernel_f64(int rows, bool own) {
  return rows == 4 ? frozen_kernel<4, true>(own) : rows == 8 ? frozen_kernel<8, true>(own) : frozen_kernel<16, true>(own);
}

}  // namespace rs
