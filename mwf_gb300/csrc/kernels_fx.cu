// Launchers of the FP64 passes in fixed point (mwf_fxpass.cuh) and of lines on their own (mwf_fxlines.cuh).
#include "mwf_fxlines.cuh"
#include "mwf_launch.h"

namespace mwf {

// Allow kernel k the most dynamic shared memory that any call of it takes.  The limit belongs to the kernel, not
// to a launch: the same value from every call keeps a launch recorded in a graph valid, and other
// threads' calls with longer lines between their own setting and launch.
template <typename K>
static cudaError_t fx_allow_smem(K k, size_t smem) {
  cudaFuncAttributes fa;
  const cudaError_t e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return e;
  const int most = (int)(zb_smem_budget(1) - fa.sharedSizeBytes);
  if (smem > (size_t)most) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

template <typename K>
static cudaError_t fx_launch(K k, int nt, const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const cudaError_t e = fx_allow_smem(k, smem);
  if (e != cudaSuccess) return e;
  k<<<n, nt, smem, st>>>(runs, items);
  return cudaGetLastError();
}

cudaError_t launch_x_forward_fx(const RunDesc* runs, const WorkItem* items, int n, size_t smem, cudaStream_t st) {
  return fx_launch(x_forward_fx_kernel, kFxForwardThreads, runs, items, n, smem, st);
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

// Lines of a CTA out of `all` that lie side by side, `outer` times: equal shares.
static int fx_line_tile(int N, int all, int most, int outer) {
  int groups = (all + most - 1) / most;
  auto tile = [&](int g) { return (all + g - 1) / g; };
  while (tile(groups) > 1 && fx_line_smem_bytes(N, tile(groups)) > zb_smem_budget(2)) ++groups;
  while (tile(groups) > 2 && (long)outer * groups < 2 * 152) ++groups;
  return tile(groups);
}

template <typename K, typename... A>
static cudaError_t fx_line_launch(K k, long grid, int N, int lines, cudaStream_t st, A... args) {
  const size_t smem = fx_line_smem_bytes(N, lines);
  const cudaError_t e = fx_allow_smem(k, smem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)grid, kFxLineThreads, smem, st>>>(args...);
  return cudaGetLastError();
}

cudaError_t launch_spec_x_backward_fx(const RunDesc* runs, int run, int MM, int KK, int NN, const void* sp, cudaStream_t st) {
  const int nb = fx_line_tile(MM, NN, 8, KK);
  const long grid = (long)KK * ((NN + nb - 1) / nb);
  const double2* in = reinterpret_cast<const double2*>(sp);
  return in ? fx_line_launch(spec_x_backward_fx_kernel<false>, grid, MM, nb, st, runs, run, nb, in)
            : fx_line_launch(spec_x_backward_fx_kernel<true>, grid, MM, nb, st, runs, run, nb, in);
}

cudaError_t launch_spec_x_forward_fx(const RunDesc* runs, int run, int MM, int KK, int NN, void* sp, cudaStream_t st) {
  const int nb = fx_line_tile(MM, NN, 8, KK);
  return fx_line_launch(spec_x_forward_fx_kernel, (long)KK * ((NN + nb - 1) / nb), MM, nb, st, runs, run, nb,
                        reinterpret_cast<double2*>(sp));
}

cudaError_t launch_phys_z_fx(const RunDesc* runs, int run, int X, int KK, int NN, double* out, cudaStream_t st) {
  const int all = (KK + 1) / 2, np = fx_line_tile(NN, all, all, X);
  return fx_line_launch(phys_z_fx_kernel, (long)X * ((all + np - 1) / np), NN, np, st, runs, run, np, out);
}

cudaError_t launch_phys_z_forward_fx(const RunDesc* runs, int run, int X, int KK, int NN, const double* ph, cudaStream_t st) {
  const int all = (KK + 1) / 2, np = fx_line_tile(NN, all, all, X);
  return fx_line_launch(phys_z_forward_fx_kernel, (long)X * ((all + np - 1) / np), NN, np, st, runs, run, np, ph);
}

cudaError_t launch_diag_z_fx(const RunDesc* runs, int run, int X, int KK, int NN, double threshold, double* out, cudaStream_t st) {
  return fx_line_launch(diag_z_fx_kernel, X, NN, (KK + 1) / 2, st, runs, run, threshold, out);
}

}  // namespace mwf
