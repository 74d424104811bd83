// Launchers of the FP64 passes in fixed point (mwf_fxpass.cuh).
#include "mwf_fxpass.cuh"
#include "mwf_launch.h"

namespace mwf {

template <typename K>
static cudaError_t fx_launch(K k, int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  // the largest size that any run takes, so that a launch recorded in a graph stays valid
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return e;
  const int most = (int)(zb_smem_budget(1) - fa.sharedSizeBytes);
  if (smem > (size_t)most) return cudaErrorInvalidValue;
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e != cudaSuccess) return e;
  k<<<n, nt, smem, st>>>(runs, items);
  return cudaGetLastError();
}

cudaError_t launch_x_forward_fx(int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  return nt == 256 ? fx_launch(x_forward_fx_kernel<256>, nt, runs, items, n, smem, st)
                   : fx_launch(x_forward_fx_kernel<512>, nt, runs, items, n, smem, st);
}

cudaError_t launch_z_fx(int K0, int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  if (K0 == 4)
    return nt == 256   ? fx_launch(z_fx_kernel<4, 256>, nt, runs, items, n, smem, st)
           : nt == 512 ? fx_launch(z_fx_kernel<4, 512>, nt, runs, items, n, smem, st)
                       : fx_launch(z_fx_kernel<4, 544>, nt, runs, items, n, smem, st);
  return nt == 256 ? fx_launch(z_fx_kernel<6, 256>, nt, runs, items, n, smem, st)
                   : fx_launch(z_fx_kernel<6, 512>, nt, runs, items, n, smem, st);
}

cudaError_t launch_x_inverse_fx(int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  return nt == 256 ? fx_launch(x_inverse_fx_kernel<256>, nt, runs, items, n, smem, st)
                   : fx_launch(x_inverse_fx_kernel<512>, nt, runs, items, n, smem, st);
}

}  // namespace mwf
