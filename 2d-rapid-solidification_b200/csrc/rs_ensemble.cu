// rs_ensemble.cu — one step of a batch of FP32 runs: column tables, tiles, the
// runs' state (rs_ensemble.cuh).
#include "rs_ens_tile.cuh"

namespace rs {
namespace {

__global__ void __launch_bounds__(kTabBlock) ens_table_kernel(const EnsRun *__restrict__ runs,
                                                              const int32_t *__restrict__ tblk) {
  pdl_wait();  // the runs' state
  pdl_trigger();
  const int32_t e = tblk[blockIdx.x];
  const EnsRun &R = runs[e >> 16];
  if (!R.active) return;
  __shared__ double kc[kTabBlock];
  table_block(R.K, ens_d0(R, R.l), R.d1, R.tab_len, R.tab, e & 0xFFFF, kc);
}

__global__ void ens_advance_kernel(EnsRun *runs, const int nruns) {
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nruns || !runs[r].active) return;
  runs[r].step += 1;
  runs[r].l += runs[r].inc_l;
}

}  // namespace

int launch_ensemble(const EnsRun *runs, int nruns, const int32_t *tblk, int ntblk, const int32_t *order, int ntiles,
                    int shape, bool advance, bool surr, int *err, cudaStream_t st) {
  if (shape < 0 || shape >= kTileShapes) return -1;
  const EnsTileKernel k = surr ? ens_net_kernel(shape) : ens_tile_of<false>(shape);
  const EnsTileFn kfn = k.fn;
  const size_t smem = k.smem;
  static std::atomic<unsigned long long> attr_done[2][kTileShapes];
  if (!smem_limit_once((const void *)kfn, (int)smem, attr_done[surr][shape])) return -3;
  static std::atomic<int> wave_of[2][kTileShapes][64];
  const int wave = resident_ctas((const void *)kfn, kThreads, smem, wave_of[surr][shape]);
  if (wave < 0) return -3;
  if (launch_dep(ens_table_kernel, dim3(ntblk), dim3(kTabBlock), st, runs, tblk) != cudaSuccess) return -3;
  // tiles scheduled while the table kernel runs share the SMs out unevenly: below
  // two waves that costs more than the launch latency it hides (us a step, tiles as
  // a dependent launch / behind the tables): 415 tiles 20.5 / 18.5, 738 22.3 / 20.5,
  // 1327 28.4 / 27.9 (490 18.5 / 20.5, 638 20.5 / 20.5); 2908 46.6 / 46.8, 3578
  // 58.5 / 59.1; with the network 415 tiles 57.2 / 53.0, 638 63.9 / 58.6
  if (ntiles < 2 * wave)
    kfn<<<ntiles, kThreads, smem, st>>>(runs, order, err, wave);
  else if (launch_dep_smem(kfn, dim3(ntiles), dim3(kThreads), smem, st, runs, order, err, wave) != cudaSuccess)
    return -3;
  if (advance && launch_dep(ens_advance_kernel, dim3((nruns + 63) / 64), dim3(64), st, const_cast<EnsRun *>(runs),
                            nruns) != cudaSuccess)
    return -3;
  return 0;
}

}  // namespace rs
