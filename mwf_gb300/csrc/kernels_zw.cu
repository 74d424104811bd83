// Launchers of the FP32 passes with a warp per line (mwf_zwarp.cuh, mwf_xwarp.cuh).
#include "mwf_xwarp.cuh"
#include "mwf_launch.h"

namespace mwf {

template <int K0, int NS, int NT, int MINB, int TW>
static cudaError_t zw_launch(const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  auto k = z_warp_kernel<K0, NS, NT, MINB, TW>;
  if (smem > zb_smem_budget(1)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zb_smem_budget(1));
  if (e != cudaSuccess) return e;
  k<<<n, NT, smem, st>>>(runs, items);
  return cudaGetLastError();
}

cudaError_t launch_z_warp(int K0, int ns, int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
#define MWF_ZW(K0_, NS_, NT_, MINB_, TW_) \
  if (K0 == K0_ && ns == NS_ && nt == NT_) return zw_launch<K0_, NS_, NT_, MINB_, TW_>(runs, items, n, smem, st);
  MWF_ZW(4, 3, 256, 2, 1) MWF_ZW(4, 3, 576, 1, 2) MWF_ZW(4, 1, 256, 2, 1) MWF_ZW(4, 1, 576, 1, 2)
  MWF_ZW(6, 3, 256, 2, 1) MWF_ZW(6, 3, 512, 1, 1) MWF_ZW(6, 1, 256, 2, 1) MWF_ZW(6, 1, 576, 1, 2)
#undef MWF_ZW
  return cudaErrorInvalidValue;
}

template <typename K>
static cudaError_t xw_launch(K k, int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (smem > zb_smem_budget(1)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zb_smem_budget(1));
  if (e != cudaSuccess) return e;
  k<<<n, nt, smem, st>>>(runs, items);
  return cudaGetLastError();
}
cudaError_t launch_x_forward_warp(int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  return nt == 256 ? xw_launch(x_forward_warp_kernel<256, 2>, nt, runs, items, n, smem, st)
                   : xw_launch(x_forward_warp_kernel<512, 1>, nt, runs, items, n, smem, st);
}
// (The x inverse waits for its update's loads: a third CTA per SM at 80 registers took 0.056 -> 0.045 ms
// on 64 M4 runs of 36 x 36; the x forward lost 15 % ... 35 % to spills there.)
cudaError_t launch_x_inverse_warp(int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  return nt == 256 ? xw_launch(x_inverse_warp_kernel<256, 3>, nt, runs, items, n, smem, st)
                   : xw_launch(x_inverse_warp_kernel<512, 1>, nt, runs, items, n, smem, st);
}

}  // namespace mwf
