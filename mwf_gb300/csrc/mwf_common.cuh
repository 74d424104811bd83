// Shared device/host definitions for the MWF timestep kernels (sm_103a).
//
// Device layouts of one run (all interleaved complex, "m" = x-wavenumber slot 0..M-1 with
// slots > MM-1 holding negative m, exactly as the reference's spectral arrays):
//   c, onl   cx<T>[NN][K][M]     MPT state and previous nonlinear term (AB2 history)
//   inv_lhs, rhs  double[NN][K][M]  FP64 implicit-update tables (1/lhs and rhs); FP32 runs
//                 hold float tables of A = rhs/lhs (hi, lo) and B = (dt/2)/lhs there (RunDesc)
//   T        cx<T>[2KK][X][NN]   x-transformed u,v,w (KK fields) and d/dx of them (KK)
//   NLT      cx<T>[KK][X][NN]    z-transformed nonlinear term, before the inverse x pass
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define MWF_MAX_STAGES 16

template <typename T> struct CxOf;
template <> struct CxOf<double> { using type = double2; };
template <> struct CxOf<float> { using type = float2; };
template <typename T> using cx = typename CxOf<T>::type;

template <typename T> __host__ __device__ __forceinline__ cx<T> mk(T a, T b) {
  cx<T> r; r.x = a; r.y = b; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// FP32: both parts in one instruction, with the same roundings.  The FP32 passes are bound by instruction
// issue more than by the FMA pipe: a step of M4 32 x 32 modes 12.8 -> 12.4 us, 1024 x 1024 2.86 -> 2.82 ms,
// M6 108 x 72 (16 runs) 0.428 -> 0.424 ms.  (Packed products and scalings gained nothing: their operands have
// to be moved into pairs.)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// a * conj(b)
template <typename C> __device__ __forceinline__ C cmulc(C a, C b) {
  C r; r.x = a.x * b.x + a.y * b.y; r.y = a.y * b.x - a.x * b.y; return r;
}
// FP32: the roundings spelled out (a fused multiply-add over one rounded product), so that every
// kernel inlining the same item code rounds alike, whatever contraction the compiler would pick
// in its context (the per-pass and the persistent FP32 kernels are compared bitwise).
template <> __device__ __forceinline__ float2 cmul<float2>(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
template <> __device__ __forceinline__ float2 cmulc<float2>(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, -__fmul_rn(a.x, b.y)));
}
// c + a b
__device__ __forceinline__ float2 cmac(float2 c, float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, __fmaf_rn(-a.y, b.y, c.x)), __fmaf_rn(a.x, b.y, __fmaf_rn(a.y, b.x, c.y)));
}
template <typename C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }

// Division by a runtime divisor 1 <= d <= 2^16 of dividends 0 <= b < 2^16:
// q = umulhi(b, ceil(2^32 / d)) is exact in that range (the rounding error of the
// reciprocal times b stays below 2^-16 <= 1/d).  All index divisions of the passes fall in
// it (dividends are bounded by a CTA's element count, at most 18 * 512).
struct FastDiv {
  unsigned m;
  int d;
  __device__ __forceinline__ int div(int b) const { return d == 1 ? b : (int)__umulhi((unsigned)b, m); }
};
// ceil(2^32 / d) for d >= 2 is floor((2^32 - 1) / d) + 1: a 32-bit division (a 64-bit one is
// a long software sequence on the device, and kernels build their divisors per thread).
__host__ __device__ inline FastDiv make_fastdiv(int d) {
  FastDiv f;
  f.d = d;
  f.m = d == 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u;
  return f;
}

// Mixed-radix Stockham plan for one line length N = 2^a 3^b.
struct FftPlanDev {
  int N;
  int nst;
  int radix[MWF_MAX_STAGES];
  int ns[MWF_MAX_STAGES];       // product of the radices of the earlier stages
  FastDiv fnb[MWF_MAX_STAGES];  // division by N / radix
  FastDiv fns[MWF_MAX_STAGES];  // division by ns
};

// Plan of the in-place transforms (mwf_fx.cuh, mwf_zwarp.cuh) for one line length N = 2^a 3^b: stage s
// has butterflies of radix[s] elements stride[s] apart, stride[s] = N / (radix[0] ... radix[s]), and
// its twiddles at tw_off[s] of the run's table, (radix - 1) stride of them.
struct FxPlan {
  int N;
  int nst;
  int radix[MWF_MAX_STAGES];
  int stride[MWF_MAX_STAGES];
  int tw_off[MWF_MAX_STAGES];
  FastDiv fnb[MWF_MAX_STAGES];  // division by N / radix
  FastDiv fst[MWF_MAX_STAGES];  // division by stride
  // mwf_zwarp.cuh: one pad element after every group of the last stage where its radix is even, so
  // that element i lies at i + i / pad, LS elements a line; in those places stage s steps by
  // step[s] within a butterfly and by bstep[s] from block to block
  FastDiv fpad;
  int LS;
  int step[MWF_MAX_STAGES];
  int bstep[MWF_MAX_STAGES];
};
constexpr int kFxMaxCols = 8;   // columns of an item of the fixed-point x passes

// Shared-memory index of element i of an FFT buffer: one pad element after every 128
// bytes, so the radix-R strided accesses of the Stockham stages spread over all banks.
template <typename T>
__host__ __device__ __forceinline__ int pad_idx(int i) { return i + (i >> (sizeof(T) == 8 ? 3 : 4)); }
template <typename T>
__host__ __device__ inline size_t padded_elems(size_t n) { return n + (n >> (sizeof(T) == 8 ? 3 : 4)) + 1; }

// Wavenumber tables of the FP64 x-forward pass (static shared memory): x positions (the
// longest x line) and columns; the host planner leaves room for them in the tile choice.
constexpr int kXTabLen = 4096;
constexpr int kXTabCols = 64;
constexpr size_t kXTabBytes = (size_t)(kXTabLen + kXTabCols) * 8;

// Per-run descriptor, resident in device memory.
struct RunDesc {
  int K0, MM, NN, M, X, Z, K, KK;
  int prec;                     // 0 = FP64, 1 = FP32
  int xf_nb;                    // columns n per x-forward work item
  int xi_nb;                    // columns n per x-inverse work item
  int z_lx;                     // x lines per z-pass work item
  int z_sum;                    // 1: each z item runs the three z-subsets of its lines and sums
                                // their outputs into the first NLT partial (FP32); 0: one subset per item
  int zb_lx;                    // x lines per item of the batched FP32 z pass (0: the run uses
                                // z_nonlinear_kernel)
  int xbf_nb, xbi_nb;           // columns per item of the subset-split FP32 x passes (0: the run
                                // uses x_forward_kernel / x_inverse_kernel)
  int xbf_items, zb_items;      // the run's x-forward and z items per step (persistent step waits)
  double alpha, gamma, dt, cth, sth, scale;
  float alpha_f, gamma_f;       // FP32 copies for the FP32 kernels (no FP64 instructions there)
  void* c;
  void* onl;
  // Implicit-update tables, computed in FP64 on the host.  FP64 runs: 1/lhs and rhs as double.
  // FP32 runs: the update is c' = A c + B (3 nl - onl); the 1/lhs slot holds A = rhs/lhs as
  // two float arrays (hi, then lo = A - hi), the rhs slot B = (dt/2)/lhs as float.
  const double* inv_lhs;
  const double* rhs;
  void* T;
  void* NLT;
  const void* twX;              // e^{-2 pi i t / X}, t < X
  const void* twQ;              // e^{-2 pi i t / NN}
  const void* twZ;              // e^{-2 pi i t / Z}
  int* nst;                     // 1 -> next step is the Euler start (reference nst flag)
  int active;                   // 0 -> the passes skip this run (a finished request)
  // Test only (mwf_test_copy_timeout): the FP32 z pass of z_nonlinear_kernel arms each staging
  // barrier with this many bytes more than its copies carry, and waits at most test_wait_ns
  // (0: about a second) for a barrier phase, so its bounded wait runs out on purpose.
  unsigned test_tx_extra;
  unsigned long long test_wait_ns;
  double diag_ct;               // threshold of the physical-space diagnostic
  FftPlanDev planX, planQ;
  // FP32 runs whose z lines a warp transforms in place (mwf_zwarp.cuh): x lines per item (0: not
  // used), plan and stage twiddles of NN
  int zw_lines;
  FxPlan zw_plan;
  const float2* zw_tw;
  // the same for the x passes (mwf_xwarp.cuh): columns per x-forward / x-inverse item (powers of two,
  // 0: not used), field and derivative at once (2) or in turn (1), plan, twiddles and element order of MM
  int xw_fnb, xw_inb, xw_nd;
  FxPlan xw_plan;
  const float2* xw_tw;
  const unsigned short* xw_rev;
  // FP64 runs in fixed point (mwf_fxpass.cuh): columns per x-forward / x-inverse item (powers of
  // two), column blocks of the x forward, x lines per z item; twiddles e^{-2 pi i t/N} as fixed-point
  // pairs (t < X, t < Z) and by stage for MM and NN; gamma n and
  // powers of alpha m as mantissa and exponent, alpha m and its square times `scale`; position ->
  // element of the digit-reversed x lines; the scales of what the passes store
  int fx;
  int fx_nb, fx_xi_nb, fx_nblk, fx_lines;
  int fx_group;                 // x lines of a warp's task in the z pass
  int fx_tab;                   // tables of NN entries that the z pass copies to shared memory: 0 ... 2
  const int4 *fx_twX, *fx_twZ, *fx_twM, *fx_twQ, *fx_gn, *fx_mp;
  const double2* fx_ms;
  const unsigned short *fx_rev, *fx_revQ;   // of the x lines, of the z lines
  int *fx_colE, *fx_blkE, *fx_rowE, *fx_minE;
  unsigned* fx_rowP;
  FxPlan fx_planM, fx_planQ;
};

// One CTA's share of a pass.
struct WorkItem {
  int run;
  int a;   // x-forward / x-inverse: first column n;  z-pass: first x line
  int b;   // x-forward: field (0..2KK-1); x-inverse: wall-normal mode k (0..K0-1); z: subset
           // 0..2, or 3 = all three summed (runs with z_sum)
  int pad; // x-forward: 1 = without the laminar base flow (diagnostics)
};

// What a call reads back, in host memory that the device writes to.
struct HostOut {
  double value;
  int flag;
  int err;
};
constexpr int kEnergyThreads = 64;   // small blocks spread a small state's FP64 operations over the SMs

// One item of the persistent FP32 step (mwf_persist.cuh): a pass work item and its kind and size,
// code = kind << 8 | size index (kinds: 0 x forward, 1 z pass of M4, 2 z pass of M6, 3 x inverse;
// size index of MM or NN in {32, 48, 64, 96, 128, 192, 256}).
struct PersistItem {
  int run, a, b, code;
};

// Device-side error bits (the kernels never trap; they record and skip).
enum {
  MWF_DERR_FFT_CAPACITY = 1,
  MWF_DERR_OUTPUT_CAPACITY = 2,
  MWF_DERR_BAD_RADIX = 4,
  MWF_DERR_COPY_TIMEOUT = 8,   // a bulk copy into shared memory did not complete within the wait limit
  MWF_DERR_WAIT_TIMEOUT = 16,  // a persistent-step item waited for its prerequisites past the limit
};
