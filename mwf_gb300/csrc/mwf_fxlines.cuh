// FP64 lines transformed on their own in 64-bit fixed point (mwf_fx.cuh; sm_103a): the stand-alone
// 2D transforms (tra_spec2phys, tra_phys2spec, transform.fftw5.f90:64-87, 126-144), the physical
// field and the physical-space diagnostics of a run.
//
// A line of 3N points is three interleaved subsets i = s + 3q of length N, as in the passes of the
// timestep.  A CTA takes the lines that lie side by side in memory -- columns n of a field in x, the
// field pairs of an x line in z -- brings their doubles to shared memory, scales each line to integers by its
// L1 norm, transforms a subset (or a short line) per warp in place, and writes rows whose
// neighbours are in the same CTA.
//
// What bounds them: latency -- a few hundred small CTAs run once.  The kernels before took one line
// to a CTA of 256 or 512 threads, of which N/12 had a butterfly, and wrote 8 of every 88 or 136 bytes:
// M6, 64 x 64 modes: x backward 47 us, z backward 119, z forward 118, x forward 47.
// Error against 80-bit arithmetic, sizes 9 ... 128: 0.3 ... 0.6 of that of the FP64-arithmetic kernels.
#pragma once
#include "mwf_fxpass.cuh"

namespace mwf {

constexpr int kFxLineThreads = 256;

// The doubles of a line wait in the places of its integers.
__device__ __forceinline__ double2 fx_raw(const longlong2* buf, int i) {
  const longlong2 v = buf[fx_at(i)];
  return make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y));
}
__device__ __forceinline__ void fx_put_raw(longlong2* buf, int i, double2 v) {
  longlong2 r;
  r.x = __double_as_longlong(v.x);
  r.y = __double_as_longlong(v.y);
  buf[fx_at(i)] = r;
}

// Exponent e with 2^extra sum(|re| + |im|) 2^e <= 2^61 over the `count` values from place `base`, by
// one warp: the largest high word first, then the sum relative to it, as in fx_row_moments.
// fine: fx_fine of the line, of which a value of a subset line is a sum of 2^(extra + 1) values backward, one forward.
__device__ __forceinline__ int fx_line_exponent(const longlong2* buf, int base, int count, int extra, const FxPlan& pl, bool inv, int& fine) {
  const int lane = threadIdx.x & 31;
  int t = 0;
  for (int i = lane; i < count; i += 32) {
    const double2 v = fx_raw(buf, base + i);
    t = max(t, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
  }
  const int top = __reduce_max_sync(0xffffffffu, t) >> 20;
  fine = 0;
  if (top == 0) return kFxZero;
  if (top >= 0x7ff) return kFxNan;
  auto part = [&](double x) {
    const int h = __double2hiint(x) & 0x7fffffff, q = h - (top - 127) * (1 << 20);
    return q < (1 << 20) || h < (1 << 20) ? 0.f : __int_as_float(q << 3);
  };
  float a = 0.f, m = 0.f;
  for (int i = lane; i < count; i += 32) {
    const double2 v = fx_raw(buf, base + i);
    const float b = part(v.x) + part(v.y);
    a += b;
    m = fmaxf(m, b);
  }
  const int e = 61 - (fx_bits_above(fx_warp_sum(a) * 1.001f) + top - 1023 + extra);
  fine = fx_fine(pl, inv, fx_warp_max(m), top - 1023 + (inv ? extra + 1 : 0), e);
  return e;
}

__device__ __forceinline__ longlong2 fx_from_double2(double2 v, int e) {
  longlong2 r;
  r.x = fx_from_double(v.x, e);
  r.y = fx_from_double(v.y, e);
  return r;
}

// Backward: the three subsets at position j from the coefficients a at j and b at j - N (none at j = 0):
// e^{2 pi i js/3N} (a + e^{-2 pi i s/3} b), om = e^{-2 pi i t/3N}.
__device__ __forceinline__ void fx_put_subsets(longlong2* buf, int base, int N, int j, longlong2 a, longlong2 b, const int4* __restrict__ om) {
  if (j == 0) {
    for (int s = 0; s < 3; ++s) buf[fx_at(base + s * N)] = a;
    return;
  }
  constexpr FxConst s3 = fx_const(kFxSqrt34);
  const i64 rx = fx_mulc(b.x, s3), ry = fx_mulc(b.y, s3);
  longlong2 h, p, q;
  h.x = a.x - fx_half(b.x);
  h.y = a.y - fx_half(b.y);
  p.x = h.x + ry; p.y = h.y - rx;
  q.x = h.x - ry; q.y = h.y + rx;
  buf[fx_at(base + j)] = cadd(a, b);
  buf[fx_at(base + N + j)] = fx_cmul<true>(p, om[j]);
  buf[fx_at(base + 2 * N + j)] = fx_cmul<true>(q, om[2 * j]);
}

// Forward: the coefficient at j (NEG: at -j) from the subsets' spectra, place p of each.
template <bool NEG>
__device__ __forceinline__ longlong2 fx_join_subsets(const longlong2* buf, int base, int N, int p, int j, const int4* __restrict__ om) {
  const longlong2 f0 = buf[fx_at(base + p)], f1 = buf[fx_at(base + N + p)], f2 = buf[fx_at(base + 2 * N + p)];
  return cadd(cadd(f0, fx_cmul<NEG>(f1, om[j])), fx_cmul<NEG>(f2, om[2 * j]));
}

// Shared memory of the line kernels: lines (odd stride, so that lanes on neighbouring lines spread
// over the banks), stage twiddles, one exponent per line.
struct FxLineSmem {
  longlong2* buf;
  int4* tw;
  int* e;
  int* fine;        // three times, for the subsets
  int* zero;        // the shift of the forward transforms' first stage
  int PS;
};
__device__ __forceinline__ FxLineSmem fx_line_smem(unsigned char* p, int N, int lines, const int4* __restrict__ stage) {
  FxLineSmem s;
  s.PS = fx_line_stride(N);
  s.buf = reinterpret_cast<longlong2*>(p);
  s.tw = reinterpret_cast<int4*>(s.buf + ((lines * s.PS + 7) & ~7));
  s.e = reinterpret_cast<int*>(s.tw + N);
  s.fine = s.e + lines;
  s.zero = s.fine + 3 * lines;
  for (int i = threadIdx.x; i < N; i += kFxLineThreads) s.tw[i] = stage[i];
  if (threadIdx.x < 3) s.zero[threadIdx.x] = 0;
  return s;
}

// All subsets of `lines` lines: a warp per subset, or per line where the three are short.
template <bool INV>
__device__ __forceinline__ void fx_line_ffts(const FxLineSmem& S, int lines, const FxPlan& pl) {
  const int per = pl.N <= 85 ? 1 : 3;
  for (int t = threadIdx.x >> 5; t < lines * per; t += kFxLineThreads / 32) {
    const int l = per == 1 ? t : t / 3;
    fx_fft<INV>(S.buf, l * S.PS + (t - l * per) * pl.N, per == 1 ? 3 : 1, pl, S.tw, INV ? nullptr : S.zero, S.fine + 3 * l, 1);
  }
}

__device__ __forceinline__ void fx_line_scale(const FxLineSmem& S, int l, int e, int g) {
  S.e[l] = e;
  for (int i = 0; i < 3; ++i) S.fine[3 * l + i] = g;
}

// x backward: field f, columns n0 ... n0 + nb - 1 of sp[n][f][ms] -> W[f][x][n].  STATE: of the
// perturbation fields of the run's state (var_mpt2spec) in the place of sp.
template <bool STATE>
__global__ void __launch_bounds__(kFxLineThreads) spec_x_backward_fx_kernel(const RunDesc* __restrict__ runs, int run, int nb,
                                                                            const double2* __restrict__ sp) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const RunDesc& R = runs[run];
  const int X = R.X, NN = R.NN, KK = R.KK, M = R.M, MM = R.MM;
  const int blocks = (NN + nb - 1) / nb, f = blockIdx.x / blocks, n0 = (blockIdx.x - f * blocks) * nb, cols = min(nb, NN - n0);
  const FxLineSmem S = fx_line_smem(smem_raw, MM, nb, R.fx_twM);
  const FastDiv f2 = make_fastdiv(2 * MM), fMM = make_fastdiv(MM);
  for (int i = threadIdx.x; i < cols * 2 * MM; i += kFxLineThreads) {
    const int l = f2.div(i), ms = i - l * 2 * MM;     // slot MM is the m = -MM that no field has
    double2 v = make_double2(0.0, 0.0);
    if (ms != MM) {
      if constexpr (STATE) {
        const int n = n0 + l, m = ms < MM ? ms : ms - 2 * MM;
        v = mpt_to_field_w<double>(R, reinterpret_cast<const double2*>(R.c), f, m, n, false, R.alpha * m, R.gamma * n,
                                   kbeta<double>(field_k(f, R.K0)));
      } else {
        v = sp[((size_t)(n0 + l) * KK + f) * M + (ms < MM ? ms : ms - 1)];
      }
    }
    fx_put_raw(S.buf, l * S.PS + ms, v);
  }
  __syncthreads();
  for (int l = threadIdx.x >> 5; l < cols; l += kFxLineThreads / 32) {
    int g;
    const int e = fx_line_exponent(S.buf, l * S.PS, 2 * MM, 0, R.fx_planM, true, g);
    if ((threadIdx.x & 31) == 0) fx_line_scale(S, l, e, g);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cols * MM; i += kFxLineThreads) {
    const int l = fMM.div(i), j = i - l * MM, base = l * S.PS;
    const int e = S.e[l] + fx_fine_bits(S.fine[3 * l]);
    const longlong2 a = fx_from_double2(fx_raw(S.buf, base + j), e);
    const longlong2 b = fx_from_double2(fx_raw(S.buf, base + MM + j), e);
    fx_put_subsets(S.buf, base, MM, j, a, b, R.fx_twX);
  }
  __syncthreads();
  fx_line_ffts<true>(S, cols, R.fx_planM);
  __syncthreads();
  double2* __restrict__ W = reinterpret_cast<double2*>(R.T) + (size_t)f * X * NN;
  const FastDiv fc = make_fastdiv(cols);
  for (int i = threadIdx.x; i < cols * X; i += kFxLineThreads) {
    const int p3 = fc.div(i), l = i - p3 * cols, s = fMM.div(p3), p = p3 - s * MM, e = S.e[l];
    const longlong2 v = S.buf[fx_at(l * S.PS + p3)];
    W[(size_t)(s + 3 * R.fx_rev[p]) * NN + n0 + l] =
        e <= kFxNan ? make_double2(nan(""), nan("")) : make_double2(fx_to_double(v.x, e), fx_to_double(v.y, e));
  }
}

// x forward: W[f][x][n] -> the kept wavenumbers of sp[n][f][ms].
__global__ void __launch_bounds__(kFxLineThreads) spec_x_forward_fx_kernel(const RunDesc* __restrict__ runs, int run, int nb,
                                                                           double2* __restrict__ sp) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const RunDesc& R = runs[run];
  const int X = R.X, NN = R.NN, KK = R.KK, M = R.M, MM = R.MM;
  const int blocks = (NN + nb - 1) / nb, f = blockIdx.x / blocks, n0 = (blockIdx.x - f * blocks) * nb, cols = min(nb, NN - n0);
  const FxLineSmem S = fx_line_smem(smem_raw, MM, nb, R.fx_twM);
  const double2* __restrict__ W = reinterpret_cast<const double2*>(R.T) + (size_t)f * X * NN;
  const FastDiv fc = make_fastdiv(cols), fMM = make_fastdiv(MM), fX = make_fastdiv(X), fM = make_fastdiv(M);
  for (int i = threadIdx.x; i < cols * X; i += kFxLineThreads) {
    const int p3 = fc.div(i), l = i - p3 * cols, s = fMM.div(p3), p = p3 - s * MM;
    fx_put_raw(S.buf, l * S.PS + p3, W[(size_t)(s + 3 * R.fx_rev[p]) * NN + n0 + l]);
  }
  __syncthreads();
  for (int l = threadIdx.x >> 5; l < cols; l += kFxLineThreads / 32) {
    int g;
    const int e = fx_line_exponent(S.buf, l * S.PS, X, 0, R.fx_planM, false, g);
    if ((threadIdx.x & 31) == 0) fx_line_scale(S, l, e, g);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < cols * X; i += kFxLineThreads) {
    const int l = fX.div(i), at = l * S.PS + i - l * X;
    S.buf[fx_at(at)] = fx_from_double2(fx_raw(S.buf, at), S.e[l] + fx_fine_bits(S.fine[3 * l]));
  }
  __syncthreads();
  fx_line_ffts<false>(S, cols, R.fx_planM);
  __syncthreads();
  for (int i = threadIdx.x; i < cols * M; i += kFxLineThreads) {
    const int l = fM.div(i), ms = i - l * M, m = signed_m(ms, MM, M), e = S.e[l];
    const longlong2 v = m >= 0 ? fx_join_subsets<false>(S.buf, l * S.PS, MM, m, m, R.fx_twX)
                               : fx_join_subsets<true>(S.buf, l * S.PS, MM, m + MM, -m, R.fx_twX);
    sp[((size_t)(n0 + l) * KK + f) * M + ms] =
        e <= kFxNan ? make_double2(nan(""), nan("")) : make_double2(fx_to_double(v.x, e), fx_to_double(v.y, e));
  }
}

// z backward of the field pairs p0 ... of x line x: the spectra a and b of two real fields make the
// line a + i b (Hermitian extension included; of n = 0 only the real part enters, as in FFTW's
// c2r).  What is left in shared memory is the two fields at z = s + 3 rev(p).
__device__ __forceinline__ void fx_z_backward(const RunDesc& R, const FxLineSmem& S, int x, int p0, int pairs) {
  const int X = R.X, NN = R.NN, KK = R.KK;
  const double2* __restrict__ T = reinterpret_cast<const double2*>(R.T);
  const FastDiv f2 = make_fastdiv(2 * NN);
  for (int i = threadIdx.x; i < pairs * 2 * NN; i += kFxLineThreads) {
    const int l = f2.div(i), r = i - l * 2 * NN, n = r < NN ? r : r - NN, f = 2 * (p0 + l) + (r >= NN);
    double2 v = f < KK ? T[((size_t)f * X + x) * NN + n] : make_double2(0.0, 0.0);
    if (n == 0) v.y = 0.0;
    fx_put_raw(S.buf, l * S.PS + r, v);
  }
  __syncthreads();
  for (int l = threadIdx.x >> 5; l < pairs; l += kFxLineThreads / 32) {
    int g;
    const int e = fx_line_exponent(S.buf, l * S.PS, 2 * NN, 1, R.fx_planQ, true, g);
    if ((threadIdx.x & 31) == 0) fx_line_scale(S, l, e, g);
  }
  __syncthreads();
  const int slots = NN / 2 + 1;                       // j and NN - j together: each needs the other's input
  const FastDiv fS = make_fastdiv(slots);
  for (int i = threadIdx.x; i < pairs * slots; i += kFxLineThreads) {
    const int l = fS.div(i), j = i - l * slots, jq = NN - j, base = l * S.PS, e = S.e[l] + fx_fine_bits(S.fine[3 * l]);
    const longlong2 a = fx_from_double2(fx_raw(S.buf, base + j), e), b = fx_from_double2(fx_raw(S.buf, base + NN + j), e);
    longlong2 u, v;
    u.x = a.x - b.y; u.y = a.y + b.x;                 // coefficient at j
    v.x = a.x + b.y; v.y = b.x - a.y;                 // coefficient at -j
    if (j == 0) {
      fx_put_subsets(S.buf, base, NN, 0, u, u, R.fx_twZ);
      continue;
    }
    const longlong2 c = fx_from_double2(fx_raw(S.buf, base + jq), e), d = fx_from_double2(fx_raw(S.buf, base + NN + jq), e);
    longlong2 uq, vq;
    uq.x = c.x - d.y; uq.y = c.y + d.x;
    vq.x = c.x + d.y; vq.y = d.x - c.y;
    fx_put_subsets(S.buf, base, NN, j, u, vq, R.fx_twZ);
    if (j != jq) fx_put_subsets(S.buf, base, NN, jq, uq, v, R.fx_twZ);
  }
  __syncthreads();
  fx_line_ffts<true>(S, pairs, R.fx_planQ);
  __syncthreads();
}

// Physical field in the reference's order (KK, 0:Z-1, 0:X-1); CTA: x line, `np` field pairs.
__global__ void __launch_bounds__(kFxLineThreads) phys_z_fx_kernel(const RunDesc* __restrict__ runs, int run, int np, double* __restrict__ out) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const RunDesc& R = runs[run];
  const int Z = R.Z, NN = R.NN, KK = R.KK, all = (KK + 1) / 2;
  const int groups = (all + np - 1) / np, x = blockIdx.x / groups, p0 = (blockIdx.x - x * groups) * np, pairs = min(np, all - p0);
  const FxLineSmem S = fx_line_smem(smem_raw, NN, np, R.fx_twQ);
  fx_z_backward(R, S, x, p0, pairs);
  const FastDiv fp = make_fastdiv(pairs), fN = make_fastdiv(NN);
  double* __restrict__ o = out + (size_t)x * Z * KK;
  for (int i = threadIdx.x; i < pairs * Z; i += kFxLineThreads) {
    const int p3 = fp.div(i), l = i - p3 * pairs, s = fN.div(p3), f = 2 * (p0 + l), e = S.e[l];
    const longlong2 v = S.buf[fx_at(l * S.PS + p3)];
    double* __restrict__ q = o + (size_t)(s + 3 * R.fx_revQ[p3 - s * NN]) * KK + f;
    q[0] = e <= kFxNan ? nan("") : fx_to_double(v.x, e);
    if (f + 1 < KK) q[1] = e <= kFxNan ? nan("") : fx_to_double(v.y, e);
  }
}

// Physical-space diagnostics of one x line: points above the threshold and the sum of the energy
// density sum of w_f v_f^2, w = 1 for the y-independent u and w, else 1/2 (velocity.f90:115-126),
// out[2x], out[2x + 1].
__global__ void __launch_bounds__(kFxLineThreads) diag_z_fx_kernel(const RunDesc* __restrict__ runs, int run, double threshold, double* __restrict__ out) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ double red[2][kFxLineThreads / 32];
  const RunDesc& R = runs[run];
  const int Z = R.Z, KK = R.KK, pairs = (KK + 1) / 2, fw = 2 * R.K0 - 1;
  const FxLineSmem S = fx_line_smem(smem_raw, R.NN, pairs, R.fx_twQ);
  fx_z_backward(R, S, blockIdx.x, 0, pairs);
  double cnt = 0.0, sum = 0.0;
  for (int z = threadIdx.x; z < Z; z += kFxLineThreads) {
    double ep = 0.0;
    for (int l = 0; l < pairs; ++l) {
      const longlong2 v = S.buf[fx_at(l * S.PS + z)];
      const int e = S.e[l], f = 2 * l;
      const double a = e <= kFxNan ? nan("") : fx_to_double(v.x, e);
      const double b = e <= kFxNan || f + 1 == KK ? 0.0 : fx_to_double(v.y, e);
      ep += (f == 0 ? 1.0 : 0.5) * a * a;
      ep += (f + 1 == fw ? 1.0 : 0.5) * b * b;
    }
    sum += ep;
    cnt += ep > threshold ? 1.0 : 0.0;
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = cnt;
    red[1][threadIdx.x >> 5] = sum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kFxLineThreads / 32; ++w) {
      cnt += red[0][w];
      sum += red[1][w];
    }
    out[2 * (size_t)blockIdx.x] = cnt;
    out[2 * (size_t)blockIdx.x + 1] = sum;
  }
}

// z forward of field pairs: physical values (KK, 0:Z-1, 0:X-1) -> W[f][x][n], times 1/(XZ).  With Y the
// spectrum of a + i b: a at n is (Y[n] + conj Y[-n]) / 2, b is (Y[n] - conj Y[-n]) / 2i.
__global__ void __launch_bounds__(kFxLineThreads) phys_z_forward_fx_kernel(const RunDesc* __restrict__ runs, int run, int np,
                                                                           const double* __restrict__ ph) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const RunDesc& R = runs[run];
  const int X = R.X, Z = R.Z, NN = R.NN, KK = R.KK, all = (KK + 1) / 2;
  const int groups = (all + np - 1) / np, x = blockIdx.x / groups, p0 = (blockIdx.x - x * groups) * np, pairs = min(np, all - p0);
  const FxLineSmem S = fx_line_smem(smem_raw, NN, np, R.fx_twQ);
  const FastDiv fp = make_fastdiv(pairs), fN = make_fastdiv(NN), fZ = make_fastdiv(Z);
  const double* __restrict__ in = ph + (size_t)x * Z * KK;
  for (int i = threadIdx.x; i < pairs * Z; i += kFxLineThreads) {
    const int p3 = fp.div(i), l = i - p3 * pairs, s = fN.div(p3), f = 2 * (p0 + l);
    const double* __restrict__ q = in + (size_t)(s + 3 * R.fx_revQ[p3 - s * NN]) * KK + f;
    fx_put_raw(S.buf, l * S.PS + p3, make_double2(q[0], f + 1 < KK ? q[1] : 0.0));
  }
  __syncthreads();
  for (int l = threadIdx.x >> 5; l < pairs; l += kFxLineThreads / 32) {
    int g;
    const int e = fx_line_exponent(S.buf, l * S.PS, Z, 0, R.fx_planQ, false, g);
    if ((threadIdx.x & 31) == 0) fx_line_scale(S, l, e, g);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < pairs * Z; i += kFxLineThreads) {
    const int l = fZ.div(i), at = l * S.PS + i - l * Z;
    S.buf[fx_at(at)] = fx_from_double2(fx_raw(S.buf, at), S.e[l] + fx_fine_bits(S.fine[3 * l]));
  }
  __syncthreads();
  fx_line_ffts<false>(S, pairs, R.fx_planQ);
  __syncthreads();
  double2* __restrict__ W = reinterpret_cast<double2*>(R.T);
  const double sc = R.scale;
  for (int i = threadIdx.x; i < pairs * NN; i += kFxLineThreads) {
    const int l = fN.div(i), n = i - l * NN, f = 2 * (p0 + l);
    const int e = S.e[l];
    const longlong2 y = fx_join_subsets<false>(S.buf, l * S.PS, NN, n, n, R.fx_twZ);
    const longlong2 q = n == 0 ? y : fx_join_subsets<true>(S.buf, l * S.PS, NN, NN - n, n, R.fx_twZ);
    auto half = [&](i64 v) { return e <= kFxNan ? nan("") : fx_to_double(v, e + 1) * sc; };
    W[((size_t)f * X + x) * NN + n] = make_double2(half(y.x + q.x), half(y.y - q.y));
    if (f + 1 < KK) W[((size_t)(f + 1) * X + x) * NN + n] = make_double2(half(y.y + q.y), half(q.x - y.x));
  }
}

}  // namespace mwf
