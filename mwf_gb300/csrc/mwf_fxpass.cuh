// The three passes of the FP64 timestep in 64-bit fixed point (mwf_fx.cuh; sm_103a).
//
//   x forward  item (run, first column n0, field f in 0 .. 2KK-1): the field's spectral values
//              (var_mpt2spec + vel_addlam + var_spec_grad, variables.f90:390-434, 600-612) as
//              integers with one scale per column, transformed in x as three interleaved subsets
//              x = s + 3q of length MM (tra_spec2phys, transform.fftw5.f90:69-78)
//   z          item (run, first x line x0, z-subset s): all NPAIR + KK backward transforms of the
//              lines z = s + 3q, the Galerkin coupling (udotgradu, modes.M4.f90:14-28 /
//              modes.M6.f90:14-20) as integer products, NPAIR forward transforms and the split
//              (transform.fftw5.f90:80-85, 126-135)
//   x inverse  item (run, first column n0, wall-normal mode k): the three partials summed, forward
//              x transforms, var_spec2mpt (variables.f90:440-480) and the update of vel_TS
//              (velocity.f90:21-41) in FP64
//
// What is stored between the passes (RunDesc, fx_*):
//   T     longlong2[2KK][X][NN], column (f, n) scaled by 2^colE[f][n]
//   rowP  unsigned[2KK][X][nblk] and blkE int[2KK][nblk]: for row (f, x) and column block b, the sum
//         and the largest of |re| + |im| over the block as two bfloat16 (rounded up; sum in the high
//         half) times 2^(32 - blkE), the last entry being column n = 0, which block 0 leaves out;
//         the z pass scales its lines by them
//   NLT   longlong2[3][KK][X][NN], row (s, f, x) scaled by 2^rowE[s][f][x]; minE[f] = the smallest
//         of field f, the scale at which the x inverse adds the partials
// Values are unnormalised; the 1/(3MM 3NN) of the forward transform is applied in the update.
#pragma once
#include "mwf_kernels.cuh"
#include "mwf_fx.cuh"
#include "nl_fx_gen.cuh"

namespace mwf {

// 2^k for k <= 0, zero below the float range.
__device__ __forceinline__ float fx_pow2(int k) { return k < -126 ? 0.f : __int_as_float((k + 127) << 23); }
// Number of bits of values whose largest high word is hi (at least 32).
__device__ __forceinline__ int fx_bitlen(int hi) { return 64 - __clz(hi); }

__device__ __forceinline__ float fx_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float fx_warp_max(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));   // v >= 0
}
// Two floats >= 0 as bfloat16, rounded up.
__device__ __forceinline__ unsigned fx_pack2(float hi, float lo) {
  return ((__float_as_uint(hi) + 0xffffu) & 0xffff0000u) | ((__float_as_uint(lo) + 0xffffu) >> 16);
}

// A sum of moduli S 2^E; S = 0: nothing but zeros.
struct FxNorm { float S; int E; };
__device__ __forceinline__ FxNorm fx_norm_add(FxNorm a, FxNorm b) {
  if (a.S == 0.f) return b;
  if (b.S == 0.f) return a;
  FxNorm r;
  r.E = max(a.E, b.E);
  r.S = a.S * fx_pow2(max(a.E - r.E, -127)) + b.S * fx_pow2(max(b.E - r.E, -127));
  return r;
}

__device__ __forceinline__ FxNorm fx_norm_mul(FxNorm a, FxNorm b) { return FxNorm{a.S * b.S, a.E + b.E}; }
// |v| (truncated by less than 2^-23; subnormals count as zero)
__device__ __forceinline__ FxNorm fx_norm(double v) {
  const u64 b = fx_bits(v);
  const int ex = (int)(b >> 52) & 0x7ff;
  return FxNorm{ex == 0 ? 0.f : __uint_as_float(0x3f800000u | ((unsigned)(b >> 29) & 0x7fffffu)), ex - 1023};
}

// ---------------------------------------------------------------------------------------
// x forward
// ---------------------------------------------------------------------------------------

// Sum and largest over the M slots of a row of |re| + |im| times |m|^p0 (S0, T0) and |m|^p1 (S1, T1),
// each as a float times 2^E; nan: a NaN or an infinity in the row.  One warp, one pass, eight loads of a lane in flight; each
// lane keeps its sums relative to its largest exponent so far.  The high words are enough (truncated
// by less than 2^-20, which the caller covers); zeros and subnormals count as zeros.
__device__ __forceinline__ void fx_row_moments(const double2* __restrict__ row, int M, int MM, int p0, int p1,
                                               float& S0, float& S1, float& T0, float& T1, int& E, int& nan) {
  const int lane = threadIdx.x & 31;
  int top = 0;
  float a = 0.f, b = 0.f, ta = 0.f, tb = 0.f;
  for (int m0 = 0; m0 < M; m0 += 256) {
    int hx[8], hy[8], t = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int ms = m0 + 32 * i + lane;
      const double2 v = ms < M ? row[ms] : make_double2(0.0, 0.0);
      hx[i] = __double2hiint(v.x) & 0x7fffffff;
      hy[i] = __double2hiint(v.y) & 0x7fffffff;
      t = max(t, max(hx[i], hy[i]));
    }
    t >>= 20;
    if (t > top) {
      const float k = fx_pow2(max(top - t, -127));
      a *= k;
      b *= k;
      ta *= k;
      tb *= k;
      top = t;
    }
    auto part = [&](int h) {                          // relative to the largest exponent
      const int q = h - (top - 127) * (1 << 20);
      return q < (1 << 20) || h < (1 << 20) ? 0.f : __int_as_float(q << 3);
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int ms = m0 + 32 * i + lane;
      const float v = part(hx[i]) + part(hy[i]);
      const float m = (float)(ms < MM ? ms : M - ms);
      const float va = v * (p0 == 0 ? 1.f : p0 == 1 ? m : p0 == 2 ? m * m : m * m * m);
      const float vb = v * (p1 == 0 ? 1.f : p1 == 1 ? m : m * m);
      a += va;
      b += vb;
      ta = fmaxf(ta, va);
      tb = fmaxf(tb, vb);
    }
  }
  const int all = __reduce_max_sync(0xffffffffu, top);
  const float k = fx_pow2(max(top - all, -127));
  S0 = fx_warp_sum(a * k);
  S1 = fx_warp_sum(b * k);
  T0 = fx_warp_max(ta * k);
  T1 = fx_warp_max(tb * k);
  E = all - 1023;
  nan = all >= 0x7ff;
}

constexpr int kFxForwardThreads = 256;   // two CTAs per SM: the widest lines fit half an SM's shared memory
__global__ void __launch_bounds__(kFxForwardThreads, 2) x_forward_fx_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  constexpr int NT = kFxForwardThreads;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  longlong2* buf = reinterpret_cast<longlong2*>(smem_raw);       // line (l, s) at (3 l + s) MM
  __shared__ int colE[kFxMaxCols];
  __shared__ FxFactor colN[2][kFxMaxCols];
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, MM = R.MM, NN = R.NN, KK = R.KK, M = R.M, K = R.K, K0 = R.K0;
  const int n0 = wi.a, f = wi.b, nbw = R.fx_nb;
  const int nb = min(nbw, NN - n0);
  const bool deriv = f >= KK;
  const int fs = deriv ? f - KK : f;
  const int k = field_k(fs, K0);
  const int comp = fs < K0 ? 0 : (fs < 2 * K0 - 1 ? 1 : 2);
  const double2* __restrict__ c = reinterpret_cast<const double2*>(R.c);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int4* tw = reinterpret_cast<int4*>(buf + ((3 * nbw * MM + 7) & ~7));
  for (int i = threadIdx.x; i < MM; i += NT) tw[i] = R.fx_twM[i];
  if (n0 == 0 && !deriv && threadIdx.x == 0) R.fx_minE[f] = 1 << 29;      // the z pass takes minima into it

  // Column scales from bounds on the columns' L1 norms: u = i(-n1 psi + k1 m1 phi), w = i(m1 psi +
  // k1 n1 phi), v = (m1^2 + n1^2) phi and the same times m1 (m1 = alpha m, n1 = gamma n)
  __shared__ float mom[2][4][kFxMaxCols];             // [psi, phi][sums, largest]
  __shared__ int fine[3 * kFxMaxCols];                // finer scale of the first stages, by subset line
  __shared__ int momE[2][kFxMaxCols], momN[2][kFxMaxCols];
  {
    const int dd = deriv ? 1 : 0;
    for (int i = warp; i < 2 * nb; i += NT / 32) {
      const int l = i >> 1, phi = i & 1;
      float s0 = 0.f, s1 = 0.f, t0 = 0.f, t1 = 0.f;
      int E = 0, bad = 0;
      // psi: u needs m^d, w m^(d+1); phi: u m^(d+1), w m^d, v m^(d+2) and m^d
      if (phi ? k >= 1 : comp != 1) {
        const int p0 = phi ? (comp == 0 ? dd + 1 : comp == 2 ? dd : dd + 2) : (comp == 0 ? dd : dd + 1);
        fx_row_moments(c + ((size_t)(n0 + l) * K + (phi ? k + K0 - 1 : k)) * M, M, MM, p0, dd, s0, s1, t0, t1, E, bad);
      }
      if (lane == 0) {
        mom[phi][0][l] = s0;
        mom[phi][1][l] = s1;
        mom[phi][2][l] = t0;
        mom[phi][3][l] = t1;
        momE[phi][l] = E;
        momN[phi][l] = bad;
      }
    }
  }
  __syncthreads();
  // (in floats with an exponent: an FP64 instruction of a warp takes 74 clocks, and these chains of
  // them were 2 us of every block)
  if (threadIdx.x < nb) {
    const int l = threadIdx.x, n = n0 + l;
    const FxNorm a1 = fx_norm(R.alpha), g1 = fx_norm_mul(fx_norm(R.gamma), FxNorm{(float)n, 0}), k1{(float)k * 1.570797f, 0};
    auto bound = [&](int i) {                         // i = 0: of the sum, 2: of the largest
      const FxNorm s0{mom[0][i][l], momE[0][l]}, t0{mom[1][i][l], momE[1][l]}, t1{mom[1][i + 1][l], momE[1][l]};
      FxNorm L = comp == 0   ? fx_norm_add(fx_norm_mul(g1, s0), fx_norm_mul(fx_norm_mul(k1, a1), t0))
                 : comp == 2 ? fx_norm_add(fx_norm_mul(a1, s0), fx_norm_mul(fx_norm_mul(k1, g1), t0))
                             : fx_norm_add(fx_norm_mul(fx_norm_mul(a1, a1), t0), fx_norm_mul(fx_norm_mul(g1, g1), t1));
      if (n == 0 && !deriv && comp != 1) {            // the mean flows u_k = psi_k, w_k = phi_k, and the base flow
        const double2 v = c[(size_t)(comp == 0 || k == 0 ? k : k + K0 - 1) * M];
        L = fx_norm_add(L, fx_norm_add(fx_norm(v.x), fx_norm(v.y)));
        if (k == 1) L = fx_norm_add(L, FxNorm{1.f, 0});
      }
      if (deriv) L = fx_norm_mul(L, a1);
      L.S *= 1.0003f;
      return L;
    };
    const FxNorm L = bound(0), most = bound(2);
    const int e = momN[0][l] || momN[1][l] ? kFxNan : (L.S == 0.f ? kFxZero : 61 - (L.E + fx_bits_above(L.S)));
    // a value of the subset lines is the sum of two coefficients
    const int fg = fx_fine(R.fx_planM, true, most.S, most.E + 1, e);
    for (int s = 0; s < 3; ++s) fine[3 * l + s] = fg;
    colE[l] = e;
    R.fx_colE[(size_t)f * NN + n] = e;
  } else if (threadIdx.x >= 32 && threadIdx.x < 32 + nb) {
    const int l = threadIdx.x - 32;
    const double n1 = R.gamma * (n0 + l), kb = kbeta<double>(k), sg = deriv ? -1.0 : 1.0;
    colN[0][l] = fx_factor(comp == 0 ? -sg * n1 : comp == 2 ? sg : 1.0);
    colN[1][l] = fx_factor(comp == 0 ? sg * kb : comp == 2 ? sg * (kb * n1) : n1 * n1);
  }
  __syncthreads();

  // fill: a = value at m = j, b = value at m = j - MM; subset s of the column has the length-MM
  // spectrum e^{2 pi i js/X} (a + e^{-2 pi i s/3} b).  A value is i^rot (A m1^pa na + B m1^pb nb) of two
  // MPT coefficients A, B, m1 = alpha m, with na, nb of the column alone:
  //   u = i (-n1 psi + k1 m1 phi),  w = i (m1 psi + k1 n1 phi),  v = (m1^2 + n1^2) phi,
  // and i m1 times that for the derivatives.  The products are integer ones on the mantissas: with
  // FP64 multiplications the fill was bound by the FP64 pipe and took 57 % of the pass.
  const int4* __restrict__ xm = R.fx_twX;             // e^{-2 pi i t/X}
  const FastDiv fMM = make_fastdiv(MM);
  const int d = deriv ? 1 : 0;
  const int pa = d + (comp == 0 ? 0 : comp == 1 ? 2 : 1), pb = d + (comp == 0 ? 1 : 0);
  const bool rot = (comp != 1) != deriv;
  const size_t rowa = (size_t)(comp == 1 ? k + K0 - 1 : k) * M, rowb = (size_t)(k + K0 - 1) * M;
  const bool hasb = k >= 1;
  const int4* __restrict__ mp = R.fx_mp;              // (alpha m)^p, p = 0 .. 3, as (h, l, exponent)
#pragma unroll 1
  for (int e = threadIdx.x; e < nb * MM; e += NT) {
    const int l = fMM.div(e);
    const int j = e - l * MM;
    const int ce = colE[l] + fx_fine_bits(fine[3 * l]);
    const FxFactor na = colN[0][l], nbf = colN[1][l];
    const double2* __restrict__ col = c + (size_t)(n0 + l) * K * M;
    const int jn = j == 0 ? 0 : MM - j;               // -m of the negative wavenumber
    const int msn = j == 0 ? 0 : M - jn;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 A = col[rowa + j], An = col[rowa + msn];
    const double2 B = hasb ? col[rowb + j] : zero, Bn = hasb ? col[rowb + msn] : zero;
    auto form = [&](double2 a, double2 b, int m, bool neg) {
      const int4 ta = mp[pa * MM + m], tb = mp[pb * MM + m];
      const FxFactor fa{ta.x, ta.y, ta.z}, fb{tb.x, tb.y, tb.z};
      i64 xa = fx_term(a.x, fa, na, ce), ya = fx_term(a.y, fa, na, ce);
      i64 xb = fx_term(b.x, fb, nbf, ce), yb = fx_term(b.y, fb, nbf, ce);
      if (neg && (pa & 1)) { xa = -xa; ya = -ya; }
      if (neg && (pb & 1)) { xb = -xb; yb = -yb; }
      longlong2 q;
      q.x = rot ? -(ya + yb) : xa + xb;
      q.y = rot ? xa + xb : ya + yb;
      return q;
    };
    longlong2 a = form(A, B, j, false);
    if (j == 0 && n0 + l == 0) {                      // mean flows: u_k = psi_k, w_k = phi_k (k >= 1), and the base flow
      double2 v = zero;
      if (!deriv && comp != 1 && k >= 1) {
        v = comp == 0 ? A : B;
        if (k == 1) v.x += comp == 0 ? R.cth : R.sth;
      }
      a.x = fx_from_double(v.x, ce);
      a.y = fx_from_double(v.y, ce);
    }
    const int base = 3 * l * MM + j;
    if (j == 0) {
      buf[fx_at(base)] = a;
      buf[fx_at(base + MM)] = a;
      buf[fx_at(base + 2 * MM)] = a;
      continue;
    }
    const longlong2 b = form(An, Bn, jn, true);
    buf[fx_at(base)] = cadd(a, b);
    constexpr FxConst s3 = fx_const(kFxSqrt34);
    const i64 rx = fx_mulc(b.x, s3), ry = fx_mulc(b.y, s3);
    longlong2 h, p, q;
    h.x = a.x - fx_half(b.x);
    h.y = a.y - fx_half(b.y);
    p.x = h.x + ry; p.y = h.y - rx;                   // a + e^{-2 pi i/3} b
    q.x = h.x - ry; q.y = h.y + rx;                   // a + e^{-4 pi i/3} b
    buf[fx_at(base + MM)] = fx_cmul<true>(p, xm[j]);
    buf[fx_at(base + 2 * MM)] = fx_cmul<true>(q, xm[2 * j]);
  }
  __syncthreads();

  {
    const int lines = 3 * nb;
    const int G = max(1, min(lines, 256 / MM));
    for (int t = warp * G; t < lines; t += (NT / 32) * G)
      fx_fft<true>(buf, t * MM, min(G, lines - t), R.fx_planM, tw, nullptr, fine + t, 1);
  }
  __syncthreads();

  // store: consecutive lanes take consecutive columns (nbw of them, a power of two), then
  // positions; the block's part of the row norms is summed over those lanes
  // (column n = 0 apart: it holds the base and mean flows, which the z derivatives do not have)
  const int nblk = R.fx_nblk, blk = n0 / nbw, lo = n0 == 0 ? 1 : 0;
  int eb = kFxZero;
  for (int l = lo; l < nb; ++l) eb = min(eb, colE[l]);
  if (threadIdx.x == 0) {
    R.fx_blkE[(size_t)f * nblk + blk] = eb;
    if (lo) R.fx_blkE[(size_t)f * nblk + nblk - 1] = colE[0];
  }
  const int lw = 31 - __clz(nbw);
  const int l = threadIdx.x & (nbw - 1);
  const bool live = l < nb, apart = l < lo;
  const int ce = live ? colE[l] : kFxZero;
  const int er = apart ? ce : eb;
  const float wgt = (ce >= kFxZero || er <= kFxNan) ? 0.f : fx_pow2(max(er - ce, -127));
  longlong2* __restrict__ T = reinterpret_cast<longlong2*>(R.T) + (size_t)f * X * NN;
  unsigned* __restrict__ P = R.fx_rowP + (size_t)f * X * nblk;
#pragma unroll 4
  for (int e0 = 0; e0 < (X << lw); e0 += NT) {
    const int sp = (e0 + threadIdx.x) >> lw;          // s MM + position
    const bool on = sp < X;
    const int s = on ? fMM.div(sp) : 0;
    const int p = on ? sp - s * MM : 0;
    const int x = s + 3 * R.fx_rev[p];
    float part = 0.f;
    if (on && live) {
      const longlong2 v = buf[fx_at((3 * l + s) * MM + p)];
      T[(size_t)x * NN + n0 + l] = v;
      part = ((float)fx_abs_hi(v.x) + (float)fx_abs_hi(v.y) + 2.f) * wgt;
    }
    if (on && apart) P[(size_t)x * nblk + nblk - 1] = fx_pack2(part, part);
    if (apart) part = 0.f;
    float top = part;
    for (int o = 1; o < nbw; o <<= 1) {
      part += __shfl_xor_sync(0xffffffffu, part, o);
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if (on && l == 0) P[(size_t)x * nblk + blk] = fx_pack2(part, top);
  }
}

// ---------------------------------------------------------------------------------------
// z pass
// ---------------------------------------------------------------------------------------

constexpr int kFxFlight = 5;   // 128 blocks and the column n = 0 are 129 entries for 32 lanes

// Sums (S) and largest (m) of the moduli of row (f, x), and of the moduli times the z wavenumber index
// (Z, mz: upper bounds with the block's largest index), times 2^E, over the W lanes (a power of two)
// of a warp's segment; lane = place in it.
struct FxRow { float S, Z, m, mz; int E, bad; };
__device__ __forceinline__ FxRow fx_row_norm(const RunDesc& R, int f, int x, int W, int lane) {
  const int nblk = R.fx_nblk;
  const unsigned* __restrict__ P = R.fx_rowP + ((size_t)f * R.X + x) * nblk;
  const int* __restrict__ EB = R.fx_blkE + (size_t)f * nblk;
  int ref = -(1 << 29);
  FxRow o{0.f, 0.f, 0.f, 0.f, 0, 0};
  for (int b0 = 0; b0 < nblk; b0 += kFxFlight * W) {  // kFxFlight blocks of a lane in flight
    unsigned p[kFxFlight];
    int e[kFxFlight], top = -(1 << 29);
#pragma unroll
    for (int i = 0; i < kFxFlight; ++i) {
      const int b = b0 + i * W + lane;
      p[i] = b < nblk ? P[b] : 0u;
      e[i] = b < nblk ? EB[b] : kFxZero;
    }
#pragma unroll
    for (int i = 0; i < kFxFlight; ++i) {
      o.bad |= e[i] <= kFxNan;
      if (p[i]) top = max(top, -e[i]);
    }
    for (int d = 1; d < W; d <<= 1) {
      top = max(top, __shfl_xor_sync(0xffffffffu, top, d));
      o.bad |= __shfl_xor_sync(0xffffffffu, o.bad, d);
    }
    if (top > ref) {                                  // the same for the whole segment
      const float k = fx_pow2(max(ref - top, -127));
      o.S *= k;
      o.Z *= k;
      o.m *= k;
      o.mz *= k;
      ref = top;
    }
#pragma unroll
    for (int i = 0; i < kFxFlight; ++i)
      if (p[i]) {
        const float k = fx_pow2(max(-e[i] - ref, -127));
        const float v = __uint_as_float(p[i] & 0xffff0000u) * k, t = __uint_as_float(p[i] << 16) * k;
        o.S += v;
        o.m = fmaxf(o.m, t);
        const int b = b0 + i * W + lane;
        if (b < nblk - 1) {                           // the last entry is n = 0
          const float n = (float)((b + 1) * R.fx_nb - 1);
          o.Z += v * n;
          o.mz = fmaxf(o.mz, t * n);
        }
      }
  }
  for (int d = 1; d < W; d <<= 1) {
    o.S += __shfl_xor_sync(0xffffffffu, o.S, d);
    o.Z += __shfl_xor_sync(0xffffffffu, o.Z, d);
    o.m = fmaxf(o.m, __shfl_xor_sync(0xffffffffu, o.m, d));
    o.mz = fmaxf(o.mz, __shfl_xor_sync(0xffffffffu, o.mz, d));
  }
  o.E = ref + 32;
  return o;
}

// Groups of values with one scale in the coupling: the velocity components, and their x and z
// derivatives.
enum { kFxU = 0, kFxV = 1, kFxW = 2, kFxDx = 3, kFxDz = 6, kFxGroups = 9 };

template <int K0> __host__ __device__ constexpr int fx_comp(int f) { return f < K0 ? 0 : (f < 2 * K0 - 1 ? 1 : 2); }
template <int K0> __host__ __device__ constexpr int fx_first(int comp) { return comp == 0 ? 0 : (comp == 1 ? K0 : 2 * K0 - 1); }
template <int K0> __host__ __device__ constexpr int fx_count(int comp) { return comp == 1 ? K0 - 1 : K0; }

template <int K0, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1) z_fx_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  constexpr int KK = 3 * K0 - 1, NPAIR = (KK + 1) / 2, NTR = NPAIR + KK;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, Q = R.NN, x0 = wi.a, s = wi.b;
  const int L = min(R.fx_lines, X - x0);
  // line (t, l) at t TS + l Q: TS is a multiple of 64, so the place of an element within the
  // lines of one t is the same for every t
  const int TS = (L * Q + 63) & ~63;
  longlong2* buf = reinterpret_cast<longlong2*>(smem_raw);
  int4* tw = reinterpret_cast<int4*>(buf + (size_t)NTR * TS);    // [Q] stage twiddles
  int* eL = reinterpret_cast<int*>(tw + Q);                      // [NTR L] line exponents
  int* mx = eL + NTR * L;                                        // [2 NTR L] the lines' finer first scale, then largest
                                                                 // high words (re, im), then shifts, then the finer scale
  int* ge = mx + 2 * NTR * L;                                    // [kFxGroups L] group exponents
  float* gb = reinterpret_cast<float*>(ge + kFxGroups * L);      // [3][kFxGroups L] of a group's fields, relative to its full
                                                                 // scale: the largest value, the sum of the
                                                                 // largest, the same sum with factors k
  int* eo = reinterpret_cast<int*>(gb + 3 * kFxGroups * L);      // [3 L] exponents of the products
  int* sh = eo + 3 * L;                                          // [NPAIR L] forward line shifts
  int* bad = sh + NPAIR * L;                                     // [L] NaN lines
  // Where they fit (RunDesc::fx_tab): the subset's twiddles e^{-2 pi i ns/Z}, then gamma n, which the fill
  // would wait for in every slot
  int4* const tab = reinterpret_cast<int4*>(smem_raw + (((unsigned char*)(bad + L) - smem_raw + 15) & ~15));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
  const longlong2* __restrict__ T = reinterpret_cast<const longlong2*>(R.T);
  const size_t fstride = (size_t)X * Q;

  const int ntab = R.fx_tab;
  for (int i = threadIdx.x; i < Q; i += NT) {
    tw[i] = R.fx_twQ[i];
    if (ntab > 0) tab[i] = R.fx_twZ[i * s];
    if (ntab > 1) tab[Q + i] = R.fx_gn[i];
  }
  for (int i = threadIdx.x; i < 2 * NTR * L; i += NT) mx[i] = 0;
  for (int i = threadIdx.x; i < L; i += NT) bad[i] = 0;
  __syncthreads();

  // ---- line scales: the rows' norms, a warp segment each (in the lines' space, not yet in use) ----
  {
    FxRow* rows = reinterpret_cast<FxRow*>(smem_raw);            // [2KK L]
    int W = 1;
    while (W < 32 && kFxFlight * W < R.fx_nblk) W <<= 1;
    const int sub = lane / W, seg = 32 / W;
    for (int i0 = warp * seg; i0 < 2 * KK * L; i0 += NW * seg) {
      const int i = min(i0 + sub, 2 * KK * L - 1);
      const int f = i / L, l = i - f * L;
      FxRow v = fx_row_norm(R, f, x0 + l, W, lane & (W - 1));
      if ((lane & (W - 1)) == 0) {
        v.Z *= fabsf(R.gamma_f);
        v.mz *= fabsf(R.gamma_f);
        rows[i] = v;
        if (v.bad) bad[l] = 1;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NTR * L; i += NT) {
      const int t = i / L, l = i - t * L;
      const bool two = t >= NPAIR || 2 * t + 1 < KK;
      const FxRow a = rows[(t < NPAIR ? 2 * t : KK + t - NPAIR) * L + l];
      const FxRow b = rows[(t < NPAIR ? 2 * t + (two ? 1 : 0) : t - NPAIR) * L + l];
      const FxNorm v = fx_norm_add(FxNorm{a.S, a.E}, FxNorm{two ? (t < NPAIR ? b.S : b.Z) : 0.f, b.E});
      const FxNorm m = fx_norm_add(FxNorm{a.m, a.E}, FxNorm{two ? (t < NPAIR ? b.m : b.mz) : 0.f, b.E});
      // the Hermitian extension doubles every coefficient: the line's norm is below 2 S 2^E, and a
      // value of a subset line is the sum of two of its coefficients
      const int e = v.S > 0.f ? 61 - (v.E + 1 + fx_bits_above(v.S * 1.001f)) : kFxZero;
      eL[i] = e;
      mx[2 * i] = fx_fine(R.fx_planQ, true, m.S, m.E + 1, e);
    }
  }
  __syncthreads();

  // ---- fill and backward transforms: a warp per line (or G short ones) ----
  // With w = e^{2 pi i ns/Z}, eps = e^{-2 pi i s/3}: H[n] = w (U + eps V) and
  // H[Q-n] = w' (U' + eps V'), w' = e^{2 pi i (Q-n)s/Z}, where U = a + i b at n, V = conj a + i conj b
  // at Q-n, and U', V' the same with n and Q-n exchanged.  Slot n < (Q+1)/2 of a line is the pair
  // (n, Q-n); slot 0 is n = 0 with, for even Q, n = Q/2 (its own partner).
  const int4* om = ntab > 0 ? tab : R.fx_twZ;         // e^{-2 pi i ns/Z} at n os
  const int os = ntab > 0 ? 1 : s;
  const int* __restrict__ colE = R.fx_colE;
  const int4* gn = ntab > 1 ? tab + Q : R.fx_gn;      // gamma n as (h, l, exponent)
  constexpr FxConst s3 = fx_const(kFxSqrt34);
  auto times_eps = [&](longlong2 a) {                 // eps a for this subset (s = 1, 2)
    const i64 rx = fx_mulc(a.x, s3), ry = fx_mulc(a.y, s3);
    longlong2 r;
    r.x = s == 1 ? -fx_half(a.x) + ry : -fx_half(a.x) - ry;
    r.y = s == 1 ? -fx_half(a.y) - rx : -fx_half(a.y) + rx;
    return r;
  };
  const int G = min(L, R.fx_group);
  const int groups = (L + G - 1) / G;
  const int slots = (Q + 1) / 2;
  const bool even = (Q & 1) == 0;
  const FastDiv fSl = make_fastdiv(slots);
  struct In { longlong2 Pa, Ra, Pb, Rb; int ea, ra, eb, rb; };
  for (int i = warp; i < NTR * groups; i += NW) {
    const int t = i / groups, l0 = (i - t * groups) * G, nl = min(G, L - l0);
    const bool der = t >= NPAIR;
    const int fa = der ? KK + t - NPAIR : 2 * t;
    const bool two = der || 2 * t + 1 < KK;
    const int fb = der ? t - NPAIR : (two ? 2 * t + 1 : fa);
    const int* __restrict__ ea = colE + (size_t)fa * Q;
    const int* __restrict__ eb = colE + (size_t)fb * Q;
    const longlong2* __restrict__ pa = T + (size_t)fa * fstride + (size_t)(x0 + l0) * Q;
    const longlong2* __restrict__ pb = T + (size_t)fb * fstride + (size_t)(x0 + l0) * Q;
    const int total = nl * slots;
    auto load = [&](int idx) {
      In v;
      const int l = fSl.div(idx), sl = idx - l * slots;
      const int n = sl ? sl : (even ? Q / 2 : 0), nq = sl ? Q - sl : 0;
      v.Pa = pa[l * Q + n];
      v.Ra = pa[l * Q + nq];
      v.Pb = pb[l * Q + n];
      v.Rb = pb[l * Q + nq];
      v.ea = ea[n]; v.ra = ea[nq]; v.eb = eb[n]; v.rb = eb[nq];
      return v;
    };
    In nx;
    if (lane < total) nx = load(lane);
    for (int idx = lane; idx < total; idx += 32) {
      const In v = nx;
      if (idx + 32 < total) nx = load(idx + 32);      // the next slot's rows while this one is formed
      const int l = fSl.div(idx), sl = idx - l * slots;
      const int n = sl ? sl : (even ? Q / 2 : 0), nq = sl ? Q - sl : n;
      const int e = eL[t * L + l0 + l] + fx_fine_bits(mx[2 * (t * L + l0 + l)]), base = t * TS + (l0 + l) * Q;
      const longlong2 Pa = fx_shift2(v.Pa, e - v.ea);
      longlong2 Ra = fx_shift2(v.Ra, e - v.ra), Pb, Rb;
      if (der) {
        // b = i gamma n f: a + i b = a - gamma n f
        const int4 gp = gn[n], gq = gn[sl ? nq : 0];
        const int sp = e - v.eb + gp.z, sq = e - v.rb + gq.z;
        Pb.x = fx_shift(fx_mulc(v.Pb.x, FxConst{gp.x, gp.y}), sp);
        Pb.y = fx_shift(fx_mulc(v.Pb.y, FxConst{gp.x, gp.y}), sp);
        Rb.x = fx_shift(fx_mulc(v.Rb.x, FxConst{gq.x, gq.y}), sq);
        Rb.y = fx_shift(fx_mulc(v.Rb.y, FxConst{gq.x, gq.y}), sq);
      } else {
        Pb = fx_shift2(v.Pb, e - v.eb);
        Rb = fx_shift2(v.Rb, e - v.rb);
        if (!two) Pb.x = Pb.y = Rb.x = Rb.y = 0;
      }
      if (sl == 0) {                                  // H = Re X_0; the z derivative has none
        longlong2 h;
        h.x = Ra.x;
        h.y = der ? 0 : Rb.x;
        buf[fx_at(base)] = h;
        Ra = Pa;
        Rb = Pb;
      }
      longlong2 U, V, U2, V2;
      if (der) {
        U.x = Pa.x - Pb.x;  U.y = Pa.y - Pb.y;
        V.x = Ra.x + Rb.x;  V.y = -Ra.y - Rb.y;
        U2.x = Ra.x - Rb.x; U2.y = Ra.y - Rb.y;
        V2.x = Pa.x + Pb.x; V2.y = -Pa.y - Pb.y;
      } else {
        U.x = Pa.x - Pb.y;  U.y = Pa.y + Pb.x;
        V.x = Ra.x + Rb.y;  V.y = Rb.x - Ra.y;
        U2.x = Ra.x - Rb.y; U2.y = Ra.y + Rb.x;
        V2.x = Pa.x + Pb.y; V2.y = Pb.x - Pa.y;
      }
      longlong2 Hn, Hq;
      if (s == 0) {
        Hn = cadd(U, V);
        Hq = cadd(U2, V2);
      } else {
        Hn = fx_cmul<true>(cadd(U, times_eps(V)), om[n * os]);
        Hq = fx_cmul<true>(cadd(U2, times_eps(V2)), om[nq * os]);
      }
      if (sl || even) buf[fx_at(base + n)] = Hn;
      if (sl) buf[fx_at(base + nq)] = Hq;
    }
    __syncwarp();
    fx_fft<true>(buf, t * TS + l0 * Q, nl, R.fx_planQ, tw, mx + 2 * (t * L + l0), mx + 2 * (t * L + l0), 2);
  }
  __syncthreads();

  // ---- one exponent per group: the largest value of a velocity group fills 58 bits, of a
  //      derivative group 59; mx becomes the shift of each part of a line to its group ----
  for (int i = threadIdx.x; i < kFxGroups * L; i += NT) {
    const int g = i / L, l = i - g * L, comp = g % 3;
    const int f0 = fx_first<K0>(comp), n = fx_count<K0>(comp);
    const bool vel = g < kFxDx;
    auto place = [&](int f) { return 2 * ((vel ? f / 2 : NPAIR + f) * L + l) + (vel ? (f & 1) : (g >= kFxDz)); };
    int top = -(1 << 29);
    for (int k = 0; k < n; ++k) top = max(top, fx_bitlen(mx[place(f0 + k)]) - eL[place(f0 + k) >> 1]);
    const int e = (vel ? 58 : 59) - top;
    ge[i] = e;
    float most = 0.f, sum = 0.f, ksum = 0.f;
    for (int k = 0; k < n; ++k) {
      const int at = place(f0 + k), r = e - eL[at >> 1];
      const float v = ((float)mx[at] + 1.f) * fx_pow2(r + 32 - (vel ? 58 : 59));
      mx[at] = r;
      most = fmaxf(most, v);
      sum += v;
      ksum += v * (float)(k + (comp == 1));
    }
    gb[i] = most;
    gb[kFxGroups * L + i] = sum;
    gb[2 * kFxGroups * L + i] = ksum;
  }
  __syncthreads();

  // ---- coupling: the projections of one component at a time, one direction after the other, so
  //      that the code of a direction is held once (straight-line code for all nine overran the
  //      instruction cache).  Where the block has three threads for a point (apart), each takes a
  //      component (a step of M4 16 x 16 modes 34.9 -> 33.3 us, 48 x 48 55.0 -> 53.3) ----
  const FastDiv fQ = make_fastdiv(Q), fLQ = make_fastdiv(L * Q);
  const size_t ts = (size_t)TS * 16;
  const bool apart = 3 * L * Q <= NT;
  // exponent of fx_sum without shifts (y: the sum is in units of b, and b/2 follows)
  auto direction = [&](int comp, int dir, int l) {
    return dir == 0   ? ge[kFxU * L + l] + ge[(kFxDx + comp) * L + l] - 60
           : dir == 1 ? ge[kFxW * L + l] + ge[(kFxDz + comp) * L + l] - 60
                      : ge[kFxV * L + l] + ge[comp * L + l] - 61;
  };
  // velocities: scaled to their group and split, in place
  for (int e = threadIdx.x; e < L * Q; e += NT) {
    const int l = L == 1 ? 0 : fQ.div(e);
    unsigned char* const at = smem_raw + (size_t)fx_at(e) * 16;
#pragma unroll
    for (int f = 0; f < KK; ++f) {
      i64* const q = reinterpret_cast<i64*>(at + (f / 2) * ts) + (f & 1);
      const FxLimbs v = fx_shift_limbs(*q, mx[2 * ((f / 2) * L + l) + (f & 1)]);
      *reinterpret_cast<int2*>(q) = make_int2(v.h, v.l);
    }
  }
  // ---- one exponent per component of the products: a bound on the three directions' sums fills 62 bits.  In a
  //      row of the coupling (i + j = k or |i - j| = k) each value of one factor meets at most two of the other, or one
  //      twice: twice the sum of the one's largest values times the other's largest bounds it.  (From the group
  //      scales and the largest weights alone the sums' rounding was five times that of their operands, and
  //      for M6 32 x 512 modes that fall by 10 from one wall-normal mode to the next the term 1.3 times as far off
  //      as with FP64 arithmetic.) ----
  for (int i = NT - 1 - threadIdx.x; i < 3 * L; i += NT) {
    const int comp = i / L, l = i - comp * L, N = kFxGroups * L;
    auto bound = [&](int s_, int d, int p) {          // groups of the factors; which sum of the second (1, or 2: factors k)
      const int a = s_ * L + l, b = d * L + l;
      const float v = p == 1 ? fminf(gb[a] * gb[N + b], gb[N + a] * gb[b]) : 1.570797f * gb[a] * gb[2 * N + b];
      return FxNorm{2.02f * v, (p == 1 ? 117 : 116) - ge[a] - ge[b]};
    };
    const FxNorm n = fx_norm_add(fx_norm_add(bound(kFxU, kFxDx + comp, 1), bound(kFxW, kFxDz + comp, 1)), bound(kFxV, comp, 2));
    int go = n.S > 0.f ? 62 - (n.E + fx_bits_above(n.S)) : 2 * kFxZero;
    for (int dir = 0; dir < 3; ++dir) go = min(go, direction(comp, dir, l) + 29);
    eo[i] = go;
  }
  __syncthreads();
  for (int e0 = 0; e0 < (apart ? 1 : L * Q); e0 += NT) {
    const int i = e0 + threadIdx.x;
    const int part = apart ? fLQ.div(i) : 0, e = i - part * (L * Q);
    const bool on = apart ? part < 3 : e < L * Q;
    const int first = on ? part : 0, last = apart ? first + 1 : 3;
    const int l = L == 1 || !on ? 0 : fQ.div(e);
    unsigned char* const at = smem_raw + (size_t)fx_at(on ? e : 0) * 16;
    auto vel = [&](int f) {
      const int2 v = *(reinterpret_cast<const int2*>(at + (f >> 1) * ts) + (f & 1));
      return FxLimbs{v.x, v.y};
    };
    constexpr FxConst b2 = fx_const(kFxQuarterPi);
#pragma unroll 1
    for (int comp = first; comp < last; ++comp) {
      const int f0 = comp == 0 ? 0 : comp == 1 ? K0 - 1 : 2 * K0 - 1;    // field of mode 0 (v has none)
      i64 sum[K0];
      FxAcc A[K0];
#pragma unroll
      for (int k = 0; k < K0; ++k) sum[k] = 0;
#pragma unroll 1
      for (int dir = on ? 0 : 3; dir < 3; ++dir) {    // x, z, y
#pragma unroll
        for (int k = 0; k < K0; ++k) A[k] = FxAcc{0, 0};
        const int up = eo[comp * L + l] - direction(comp, dir, l);
        if (dir < 2) {
          FxLimbs S[K0];
          const int s0 = dir ? 2 * K0 - 1 : 0;
#pragma unroll
          for (int k = 0; k < K0; ++k) S[k] = vel(s0 + k);
          auto ld = [&](int j) {
            const i64 q = *(reinterpret_cast<const i64*>(at + (NPAIR + f0 + j) * ts) + dir);
            return fx_shift_limbs(q, mx[2 * ((NPAIR + f0 + j) * L + l) + dir]);
          };
          if constexpr (K0 == 4) { if (comp == 1) nl_fx_v_4(S, ld, A); else nl_fx_p_4(S, ld, A); }
          else { if (comp == 1) nl_fx_v_6(S, ld, A); else nl_fx_p_6(S, ld, A); }
        } else {
          // in units of b = pi/2: 2 nl = sum v (j f_j) b
          FxLimbs V[K0], F[K0];
          V[0] = F[0] = FxLimbs{0, 0};
#pragma unroll
          for (int k = 1; k < K0; ++k) V[k] = vel(K0 - 1 + k);
          if (comp != 1) {
#pragma unroll
            for (int k = 1; k < K0; ++k) F[k] = vel(f0 + k);
            if constexpr (K0 == 4) nl_fx_yp_4(V, F, A); else nl_fx_yp_6(V, F, A);
          } else {
            if constexpr (K0 == 4) nl_fx_yv_4(V, A); else nl_fx_yv_6(V, A);
          }
        }
        // to the component's exponent: up by less than 30 bits, or down (a direction far below the others)
        i64 x[K0];
#pragma unroll
        for (int k = 0; k < K0; ++k) x[k] = fx_sum(A[k], max(up, 0));
        if (up < 0) {
          const int r = min(-up, 62);
#pragma unroll
          for (int k = 0; k < K0; ++k) x[k] = fx_down(x[k] << 1, r + 1);
        }
        if (dir == 2) {
#pragma unroll
          for (int k = 0; k < K0; ++k) x[k] = fx_mulc(x[k], b2);
        }
#pragma unroll
        for (int k = 0; k < K0; ++k) sum[k] += x[k];
      }
      // field f goes to line NPAIR + f/2, where only derivatives of this or an earlier component were
      if (apart) __syncthreads();
      if (!on) continue;
#pragma unroll
      for (int k = 0; k < K0; ++k) {
        if (comp == 1 && k == 0) continue;
        const int f = f0 + k;
        *(reinterpret_cast<i64*>(at + (NPAIR + (f >> 1)) * ts) + (f & 1)) = sum[k];
      }
    }
    if ((KK & 1) && on && last == 3) *(reinterpret_cast<i64*>(at + (NPAIR + KK / 2) * ts) + 1) = 0;
  }
  __syncthreads();

  // ---- forward transforms, split and store ----
  longlong2* __restrict__ NLT = reinterpret_cast<longlong2*>(R.NLT) + (size_t)s * KK * fstride;
  int WQ = 1;
  while (WQ < 32 && WQ < Q) WQ <<= 1;
  for (int i = warp; i < NPAIR * groups; i += NW) {
    const int t = i / groups, l0 = (i - t * groups) * G, nl = min(G, L - l0);
    const int first = (NPAIR + t) * TS + l0 * Q;
    // scale each line so that its norm just fits (from the high words, rounded up)
    for (int l = lane / WQ; l - lane / WQ < nl; l += 32 / WQ) {
      float a = 0.f, m = 0.f;
      if (l < nl)
        for (int n = lane & (WQ - 1); n < Q; n += WQ) {
          const longlong2 v = buf[fx_at(first + l * Q + n)];
          const float b = (float)fx_abs_hi(v.x) + (float)fx_abs_hi(v.y) + 2.f;
          a += b;
          m = fmaxf(m, b);
        }
      for (int o = 1; o < WQ; o <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      }
      if (l < nl && (lane & (WQ - 1)) == 0) {
        const int i = t * L + l0 + l, e = 61 - 32 - fx_bits_above(a * 1.001f), g = fx_fine(R.fx_planQ, false, m, 32, e);
        sh[i] = e + fx_fine_bits(g);
        mx[2 * i] = g;
      }
    }
    __syncwarp();
    fx_fft<false>(buf, first, nl, R.fx_planQ, tw, sh + t * L + l0, mx + 2 * (t * L + l0), 2);
    const int ka = 2 * t;
    const bool two = ka + 1 < KK;
    longlong2* __restrict__ oa = NLT + (size_t)ka * fstride + (size_t)(x0 + l0) * Q;
    longlong2* __restrict__ ob = oa + fstride;
    // A = G[n] + conj G[Q-n] and B = (G[n] - conj G[Q-n]) / i are twice the spectra at n; at Q-n
    // they are conj(A), conj(B), and e^{-2 pi i (Q-n)s/Z} = eps conj(e^{-2 pi i ns/Z})
    for (int idx = lane; idx < nl * slots; idx += 32) {
      const int l = fSl.div(idx), sl = idx - l * slots;
      const int base = first + l * Q, o = l * Q;
      const int n = sl ? sl : (even ? Q / 2 : 0), nq = sl ? Q - sl : n;
      const longlong2 g = buf[fx_at(base + n)], m = buf[fx_at(base + nq)];
      longlong2 A, B;
      A.x = g.x + m.x; A.y = g.y - m.y;
      B.x = g.y + m.y; B.y = m.x - g.x;
      if (s != 0) {
        const int4 w = om[n * os];
        A = fx_cmul<false>(A, w);
        B = fx_cmul<false>(B, w);
      }
      if (sl || even) {
        oa[o + n] = A;
        if (two) ob[o + n] = B;
      }
      if (sl) {
        A.y = -A.y;
        B.y = -B.y;
        if (s != 0) { A = times_eps(A); B = times_eps(B); }
        oa[o + nq] = A;
        if (two) ob[o + nq] = B;
      } else {
        const longlong2 z = buf[fx_at(base)];
        A.x = 2 * z.x; A.y = 0;
        B.x = 2 * z.y; B.y = 0;
        oa[o] = A;
        if (two) ob[o] = B;
      }
    }
    for (int j = lane; j < nl * 2; j += 32) {
      const int l = l0 + (j >> 1), f = ka + (j & 1);
      if (f >= KK) continue;
      // the coupling is 2 nl, the split another factor of two
      int e = eo[fx_comp<K0>(f) * L + l] + sh[t * L + l] - fx_fine_bits(mx[2 * (t * L + l)]) + 2;
      if (bad[l]) e = kFxNan;
      R.fx_rowE[((size_t)s * KK + f) * X + x0 + l] = e;
      atomicMin(&R.fx_minE[f], e);
    }
  }
}

// ---------------------------------------------------------------------------------------
// x inverse and update
// ---------------------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) x_inverse_fx_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  longlong2* buf = reinterpret_cast<longlong2*>(smem_raw);       // line (comp, l, s) at ((comp nb + l) 3 + s) MM
  __shared__ u64 norm[9 * kFxMaxCols];
  __shared__ int sh[9 * kFxMaxCols];
  __shared__ int fine[9 * kFxMaxCols];                // largest values' bits, then the finer scale of the first stages
  __shared__ double colw[3][kFxMaxCols];              // gamma n, (-1)^k k b gamma n and (gamma n)^2, times the scale
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, MM = R.MM, NN = R.NN, M = R.M, K0 = R.K0, K = R.K, KK = R.KK;
  const int n0 = wi.a, k = wi.b, nbw = R.fx_xi_nb;
  const int nb = min(nbw, NN - n0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
  const longlong2* __restrict__ NLT = reinterpret_cast<const longlong2*>(R.NLT);
  const size_t fstride = (size_t)X * NN;
  const int fu = k, fv = K0 + k - 1, fw = 2 * K0 - 1 + k;
  const FastDiv fMM = make_fastdiv(MM);
  int4* tw = reinterpret_cast<int4*>(buf + ((9 * nbw * MM + 7) & ~7));
  for (int i = threadIdx.x; i < MM; i += NT) tw[i] = R.fx_twM[i];
  if (threadIdx.x < nb) {
    const double n1 = R.gamma * (n0 + threadIdx.x), n1s = n1 * R.scale;
    colw[0][threadIdx.x] = n1s;
    colw[1][threadIdx.x] = kbeta<double>(k) * n1s;
    colw[2][threadIdx.x] = n1 * n1s;
  }
  const int lw = 31 - __clz(nbw);
  const int l_ = threadIdx.x & (nbw - 1);
  int ref[3];                                         // scale of each field's sum of partials
#pragma unroll
  for (int comp = 0; comp < 3; ++comp)
    ref[comp] = (comp == 1 && k == 0) ? kFxZero : R.fx_minE[comp == 0 ? fu : comp == 1 ? fv : fw] - 2;

  // load: consecutive lanes take consecutive columns, then positions
  if (l_ < nb) {
    for (int comp = 0; comp < 3; ++comp) {
      const int f = comp == 0 ? fu : comp == 1 ? fv : fw;
      const bool none = comp == 1 && k == 0;
      for (int sp = threadIdx.x >> lw; sp < X; sp += NT >> lw) {
        const int s = fMM.div(sp), p = sp - s * MM;
        longlong2 v;
        v.x = v.y = 0;
        if (!none) {
          const int x = s + 3 * R.fx_rev[p];
          const size_t o = (size_t)f * fstride + (size_t)x * NN + n0 + l_;
          const size_t ss = (size_t)KK * fstride;
          const int* __restrict__ E = R.fx_rowE + (size_t)f * X + x;
#pragma unroll
          for (int z = 0; z < 3; ++z) {
            const longlong2 q = NLT[o + z * ss];
            const int r = E[(size_t)z * KK * X] - ref[comp];     // at least 2
            v.x += fx_down(q.x, r);
            v.y += fx_down(q.y, r);
          }
        }
        buf[fx_at(((comp * nb + l_) * 3 + s) * MM + p)] = v;
      }
    }
  }
  __syncthreads();
  for (int i = warp; i < 9 * nb; i += NW) {
    u64 a = 0, m = 0;
    for (int p = lane; p < MM; p += 32) {
      const longlong2 v = buf[fx_at(i * MM + p)];
      const u64 b = ((u64)(v.x ^ (v.x >> 63)) >> 13) + ((u64)(v.y ^ (v.y >> 63)) >> 13) + 2;
      a += b;
      m |= b;                                         // an upper bound by less than a factor of two
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(m >> 32)), lo = __reduce_or_sync(0xffffffffu, (unsigned)m);
    if (lane == 0) {
      norm[i] = a;
      fine[i] = hi ? 64 - __clz((int)hi) : 32 - __clz((int)lo);
    }
  }
  __syncthreads();
  // the three subsets of a line share a scale: their combined norm is below 2^61
  for (int i = threadIdx.x; i < 9 * nb; i += NT) {
    const int b = i / 3 * 3;
    sh[i] = 61 - 13 - (64 - __clzll((i64)(norm[b] + norm[b + 1] + norm[b + 2])));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * nb; i += NT) {
    const int most = max(fine[3 * i], max(fine[3 * i + 1], fine[3 * i + 2]));
    const int g = fx_fine(R.fx_planM, false, 1.f, most + 13, sh[3 * i]);
    for (int s = 0; s < 3; ++s) {
      fine[3 * i + s] = g;
      sh[3 * i + s] += fx_fine_bits(g);
    }
  }
  __syncthreads();
  {
    const int lines = 9 * nb;
    const int G = max(1, min(lines, 256 / MM));
    for (int t = warp * G; t < lines; t += NW * G)
      fx_fft<false>(buf, t * MM, min(G, lines - t), R.fx_planM, tw, sh + t, fine + t, 1);
  }
  __syncthreads();

  const int4* __restrict__ xm = R.fx_twX;
  double2* __restrict__ c = reinterpret_cast<double2*>(R.c);
  double2* __restrict__ onl = reinterpret_cast<double2*>(R.onl);
  // The wavenumbers carry the 1/(3MM 3NN) of the transforms and come from tables: forming them in place
  // (conversions, products, the scale) made 44 FP64 operations per mode, which bound the pass.
  const double* __restrict__ ilhs = R.inv_lhs;
  const double* __restrict__ rhs = R.rhs;
  const double hdt = R.dt / 2.0;
  const double2* __restrict__ mtab = R.fx_ms;         // (alpha m, (alpha m)^2) times the scale
  const bool first = *R.nst != 0;
  const double kb1 = kbeta<double>(k);
  const FastDiv fM = make_fastdiv(M);
#pragma unroll 1
  for (int o = threadIdx.x; o < nb * M; o += NT) {
    const int l = fM.div(o);
    const int ms = o - l * M;
    const int n = n0 + l;
    const double n1 = colw[0][l], kn = colw[1][l], n2 = colw[2][l];
    auto scale = [&](int c) { return ref[c] + sh[(c * nb + l) * 3] - fx_fine_bits(fine[(c * nb + l) * 3]); };
    const int eu = scale(0), ev = scale(1), ew = scale(2);
    const int m = signed_m(ms, MM, M);
    const size_t i0 = ((size_t)n * K + k) * M + ms;
    const size_t i1 = i0 + (size_t)(K0 - 1) * M;
    const double2 zero = make_double2(0.0, 0.0);
    // operands of both slots first, so that their loads overlap the rest
    const double2 c0 = c[i0], o0 = onl[i0];
    const double r0 = rhs[i0], v0 = ilhs[i0];
    const double2 c1 = k > 0 ? c[i1] : zero, o1 = k > 0 ? onl[i1] : zero;
    const double r1 = k > 0 ? rhs[i1] : 0.0, v1 = k > 0 ? ilhs[i1] : 0.0;
    const double2 mt = mtab[m < 0 ? -m : m];
    const int j = m >= 0 ? m : m + MM;
    const int4 w1 = xm[m >= 0 ? m : m + X], w2 = xm[m >= 0 ? 2 * m : 2 * m + X];
    auto comp = [&](int i, int e, bool bad) {
      const int base = (i * nb + l) * 3 * MM + j;
      const longlong2 F0 = buf[fx_at(base)], F1 = buf[fx_at(base + MM)], F2 = buf[fx_at(base + 2 * MM)];
      const longlong2 v = cadd(cadd(F0, fx_cmul<false>(F1, w1)), fx_cmul<false>(F2, w2));
      return bad ? make_double2(nan(""), nan("")) : make_double2(fx_to_double(v.x, e), fx_to_double(v.y, e));
    };
    const double2 su = comp(0, eu, ref[0] < kFxNan / 2), sw = comp(2, ew, ref[2] < kFxNan / 2);
    const double2 sv = k > 0 ? comp(1, ev, ref[1] < kFxNan / 2) : zero;
    const double m1 = m < 0 ? -mt.x : mt.x, km = kb1 * m1, H = mt.y + n2;
    // var_spec2mpt (variables.f90:455-464)
    double2 nphi, npsi;
    nphi.x = -fma(su.y, km, fma(sw.y, kn, sv.x * H));
    nphi.y = fma(su.x, km, fma(sw.x, kn, -(sv.y * H)));
    npsi.x = fma(sw.y, m1, -(su.y * n1));
    npsi.y = fma(-sw.x, m1, su.x * n1);
    if (ms == 0 && n == 0) {   // mean modes (variables.f90:467-479)
      if (k == 0) npsi = zero;
      else {
        npsi = make_double2(-su.x * R.scale, -su.y * R.scale);
        nphi = make_double2(-sw.x * R.scale, -sw.y * R.scale);
      }
    }
    // AB2 / implicit update (velocity.f90:24-40); onl <- nl
    // (rounded as the FP64-arithmetic pass rounds it: rr c first, which is nearly all of the sum)
    auto update = [&](double rr, double il, double cv, double nv, double ov) {
      return fma(hdt, fma(3.0, nv, -ov), __dmul_rn(rr, cv)) * il;
    };
    {
      const double2 ov = first ? npsi : o0;
      double x = update(r0, v0, c0.x, npsi.x, ov.x);
      const double y = update(r0, v0, c0.y, npsi.y, ov.y);
      if (k == 0 && ms == 0 && n == 0) x = 0.0;
      c[i0] = make_double2(x, y);
      onl[i0] = npsi;
    }
    if (k > 0) {
      const double2 ov = first ? nphi : o1;
      c[i1] = make_double2(update(r1, v1, c1.x, nphi.x, ov.x), update(r1, v1, c1.y, nphi.y, ov.y));
      onl[i1] = nphi;
    }
  }
}

}  // namespace mwf
