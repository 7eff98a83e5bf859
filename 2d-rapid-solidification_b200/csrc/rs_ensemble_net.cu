// rs_ensemble_net.cu — the ensemble's tile kernels through the learned network.
#include "rs_ens_tile.cuh"

namespace rs {

EnsTileKernel ens_net_kernel(int shape) { return ens_tile_of<true>(shape); }

}  // namespace rs
