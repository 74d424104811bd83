// 64-bit fixed-point transforms of the FP64 passes (sm_103a).
//
// GB300 issues 1.74 FP64 operations per clock and SM and 57 64-bit integer additions (both
// measured), and an FFT is mostly additions.  So the FP64 passes hold the lines that they transform
// as 64-bit integers q = x 2^e with one exponent e per line: additions are exact, a product with
// a twiddle rounds once at 2^-62 of the operand's scale.  The exponent comes from the line's
// L1 norm (the sum of its moduli is at most 2^61), which bounds every partial sum of the
// transform, so nothing overflows.  A rounding early in the transform counts most: with N
// coefficients alike the L1 norm is about 1.6 N of them, so 2^-61 of it is 2^-50 of a coefficient at
// N = 1024, more than the 2^-53 of FP64 arithmetic.  So until the first two stages are
// done, whose results are sums of only a few values, a line has finer scales from its largest value
// (fx_fine).  Error of the nonlinear term against extended precision, lengths of 3 ... 1024 modes,
// as a fraction of that of the FP64-arithmetic kernels: Gaussian states 0.16 ... 0.31 on square grids and up to 0.95 on
// thin ones, spectra 1 / (1 + k^2 / 20) 0.36 ... 0.92, white ones 0.27 ... 0.86, wall-normal modes that fall by 10 from
// one to the next 0.4 ... 1.07 (of the whole term; the last of such modes alone up to 50: the coupling's operands share a
// scale).
//
// Transforms are in place, decimation in frequency backward (natural in, digit-reversed out) and
// decimation in time forward (digit-reversed in, natural out): a butterfly reads and writes the
// same elements, so one warp transforms a line (or a few short ones) with a warp barrier per stage
// and no second buffer, and the pointwise product between the two does not care about the order.
#pragma once
#include "mwf_common.cuh"

namespace mwf {

typedef long long i64;
typedef unsigned long long u64;

// Exponents: of an all-zero line (any shift of it gives zero), and of a line with a NaN or an
// infinity (the values made from it are NaN).
constexpr int kFxZero = 1 << 20;
constexpr int kFxNan = -(1 << 28);

// A constant or twiddle w 2^62 = h 2^32 + l, l in [-2^31, 2^31).
struct FxConst { int h, l; };
__host__ __device__ constexpr FxConst fx_const(i64 w) {
  return FxConst{(int)((w - (i64)(int)(unsigned)(w & 0xffffffffll)) >> 32), (int)(unsigned)(w & 0xffffffffll)};
}
constexpr i64 kFxSqrtHalf = 3260954456333195553ll;   // sqrt(1/2) 2^62
constexpr i64 kFxSqrt34 = 3993837246235628775ll;     // sqrt(3)/2
constexpr i64 kFxQuarterPi = 3622009729038561421ll;  // pi/4
// cos and sin of 2 pi k/9 for k = 1, 2, 4 (i = 0, 1, 2)
__host__ __device__ constexpr i64 fx_c9(int i) { return i == 0 ? 3532756447825785444ll : i == 1 ? 800810873071977681ll : -4333567320897763126ll; }
__host__ __device__ constexpr i64 fx_s9(int i) { return i == 0 ? 2964334632409774423ll : i == 1 ? 4541624145405292212ll : 1577289512995517789ll; }

// a b + c.  (Written as one instruction: from (i64)a * b + c the compiler made a product and an
// addition where it saw sums of several, and a coupling section of 54 such triples took 4180 cycles
// instead of 2570.)
__host__ __device__ __forceinline__ i64 fx_madw(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (i64)a * b + c;
#endif
}

// x = h 2^32 + l with l signed.
__host__ __device__ __forceinline__ FxConst fx_split(i64 x) {
  FxConst o;
  o.l = (int)(unsigned)(u64)x;
  o.h = (int)((u64)x >> 32) + (int)((unsigned)o.l >> 31);
  return o;
}
// (hi 2^64 + cross 2^32) / 2^62: the top of a product sum, cross already holding the rounding half.
__host__ __device__ __forceinline__ i64 fx_top(i64 hi, i64 cross) { return (i64)((u64)hi << 2) | (i64)((unsigned)(u64)cross >> 30); }
constexpr i64 kFxHalf = 1ll << 29;

// x w, |x| <= 2^62, rounded; the product of the low halves (below a quarter of the last bit) is dropped.
__host__ __device__ __forceinline__ i64 fx_mulc(i64 x, FxConst w) {
  const FxConst a = fx_split(x);
  const i64 cr = fx_madw(a.h, w.l, fx_madw(a.l, w.h, kFxHalf));
  return fx_top(fx_madw(a.h, w.h, (i64)(int)(cr >> 32)), cr);
}
// a w (CONJ: a conj(w)), |a| <= 2^62, twiddle w = {re h, re l, im h, im l} with low parts above -2^31.
template <bool CONJ>
__host__ __device__ __forceinline__ longlong2 fx_cmul(longlong2 a, int4 w) {
  const FxConst x = fx_split(a.x), y = fx_split(a.y);
  const int ph = CONJ ? -w.z : w.z, pl = CONJ ? -w.w : w.w;
  const int nh = CONJ ? w.z : -w.z, nl = CONJ ? w.w : -w.w;
  const i64 c1 = fx_madw(x.h, w.y, fx_madw(x.l, w.x, fx_madw(y.h, nl, fx_madw(y.l, nh, kFxHalf))));
  const i64 c2 = fx_madw(x.h, pl, fx_madw(x.l, ph, fx_madw(y.h, w.y, fx_madw(y.l, w.x, kFxHalf))));
  longlong2 r;
  r.x = fx_top(fx_madw(x.h, w.x, fx_madw(y.h, nh, (i64)(int)(c1 >> 32))), c1);
  r.y = fx_top(fx_madw(x.h, ph, fx_madw(y.h, w.x, (i64)(int)(c2 >> 32))), c2);
  return r;
}

// Shifts by any amount (64 and more shift everything out).
__host__ __device__ __forceinline__ i64 fx_shl(i64 x, int k) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(k));
  return r;
#else
  return k > 63 ? 0 : (i64)((u64)x << k);
#endif
}
__host__ __device__ __forceinline__ i64 fx_sar(i64 x, int k) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(k));
  return r;
#else
  return x >> (k > 63 ? 63 : k);
#endif
}
// x 2^sh for |x| < 2^62, rounded to nearest when sh < 0; sh may be any integer (left shifts are
// bounded by the caller's scale, or x = 0).
__host__ __device__ __forceinline__ i64 fx_shift(i64 x, int sh) {
  const int up = sh > 0 ? sh : 0;
  return (fx_sar(fx_shl(x, up + 1), up - sh) + 1) >> 1;
}
// x 2^-r, r >= 1, |x| <= 2^62, and x / 2, rounded to nearest, ties to even: ties rounded up are a bias of 2^-(r+1),
// the same for all values of a stage, which the later stages add up in the lowest wavenumbers (M4
// 512 x 512, white spectrum: the nonlinear term was 1.24 times as far off as with FP64 arithmetic, with ties
// to even 0.96 and, the coupling's sums rounded more finely, 0.47).
// Shifts beyond 63, which leave nothing, are those of 63 (of 64 and more the half of the last bit
// would be 0 or overflow, and everything, zeros too, could become -1): they come from directions or
// rows of the coupling that are zero, or far below the others.
__host__ __device__ __forceinline__ i64 fx_down(i64 x, int r) {
  const int k = r < 63 ? r : 63;
  return fx_sar(x + (fx_shl(1, k - 1) - 1) + (i64)((int)fx_sar(x, k) & 1), k);
}
__host__ __device__ __forceinline__ i64 fx_half(i64 x) { return (x >> 1) + (i64)((int)x & (int)(x >> 1) & 1); }
__host__ __device__ __forceinline__ longlong2 fx_shift2(longlong2 a, int sh) {
  longlong2 r;
  r.x = fx_shift(a.x, sh);
  r.y = fx_shift(a.y, sh);
  return r;
}

__host__ __device__ __forceinline__ u64 fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  union { double d; u64 u; } v;
  v.d = x;
  return v.u;
#endif
}
__host__ __device__ __forceinline__ double fx_value(u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)b);
#else
  union { double d; u64 u; } v;
  v.u = b;
  return v.d;
#endif
}
// round(x 2^e), |x| 2^e <= 2^61; subnormals, infinities and NaNs give values nothing reads (their
// line's exponent says so).
__host__ __device__ __forceinline__ i64 fx_from_double(double x, int e) {
  const u64 b = fx_bits(x);
  const int ex = (int)(b >> 52) & 0x7ff;
  const u64 m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
  const int r = 1085 - ex - e;
  i64 q = (i64)(((m >> ((r < 1 ? 1 : r > 63 ? 63 : r) - 1)) + 1) >> 1);
  if (ex == 0 || r > 63) q = 0;
  return (i64)b < 0 ? -q : q;
}
// q 2^-e as a double, rounded; past the double range to 0 or infinity.
__host__ __device__ __forceinline__ double fx_to_double(i64 q, int e) {
  if (q == 0) return 0.0;
  const u64 a = q < 0 ? 0ull - (u64)q : (u64)q;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((i64)a);
#else
  const int lz = __builtin_clzll(a);
#endif
  const u64 m = a << lz;
  const int field = 1023 + 63 - lz - e;
  u64 b = ((u64)(unsigned)(field - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
  if (field <= 0) b = 0;
  if (field >= 2047) b = 0x7ffull << 52;
  return fx_value(b | (q < 0 ? 0x8000000000000000ull : 0ull));
}

// A factor w = (h 2^32 + l) 2^(e - 62) with the mantissa in [1/2, 1) (zero: h = l = 0).
struct FxFactor { int h, l, e; };
__host__ __device__ __forceinline__ FxFactor fx_factor(double w) {
  const u64 b = fx_bits(w);
  const int ex = (int)(b >> 52) & 0x7ff;
  i64 m = (i64)(((b & 0xfffffffffffffull) | 0x10000000000000ull) << 9);
  if ((i64)b < 0) m = -m;
  if (ex == 0) m = 0;
  const FxConst c = fx_split(m);
  return FxFactor{c.h, c.l, ex - 1022};
}
// round(x m n 2^e) for factors m, n; |.| <= 2^61.  Two integer products on the mantissa in the place
// of FP64 multiplications.
__host__ __device__ __forceinline__ i64 fx_term(double x, FxFactor m, FxFactor n, int e) {
  const u64 b = fx_bits(x);
  const int ex = (int)(b >> 52) & 0x7ff;
  i64 v = (i64)(((b & 0xfffffffffffffull) | 0x10000000000000ull) << 9);
  v = fx_mulc(fx_mulc(v, FxConst{m.h, m.l}), FxConst{n.h, n.l});
  v = fx_shift(v, ex - 1084 + m.e + n.e + e);
  if (ex == 0) v = 0;
  return (i64)b < 0 ? -v : v;
}

// Element index -> place: the low three bits (16-byte columns of a 128-byte row) are mixed with
// the row, so strided butterflies spread over the banks without padding.
__device__ __forceinline__ int fx_at(int i) { return i ^ ((i >> 3) & 7); }

// ---- butterflies: INV = e^{+i}, otherwise e^{-i} ----
template <bool INV> __device__ __forceinline__ longlong2 fx_rot(longlong2 a) {   // times +-i
  longlong2 r;
  if (INV) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}
template <bool INV> __device__ __forceinline__ longlong2 fx_w8(longlong2 a) {    // times e^{+-i pi/4}
  constexpr FxConst h = fx_const(kFxSqrtHalf);
  longlong2 r;
  if (INV) { r.x = fx_mulc(a.x - a.y, h); r.y = fx_mulc(a.x + a.y, h); }
  else     { r.x = fx_mulc(a.x + a.y, h); r.y = fx_mulc(a.y - a.x, h); }
  return r;
}
template <bool INV> __device__ __forceinline__ void fx_dft3(longlong2& a, longlong2& b, longlong2& c) {
  constexpr FxConst s = fx_const(kFxSqrt34);
  const longlong2 t1 = cadd(b, c), t2 = csub(b, c);
  longlong2 m, j;
  m.x = a.x - fx_half(t1.x);
  m.y = a.y - fx_half(t1.y);
  j.x = fx_mulc(t2.y, s);
  j.y = fx_mulc(t2.x, s);
  if (INV) j.x = -j.x; else j.y = -j.y;
  a = cadd(a, t1);
  b = cadd(m, j);
  c = csub(m, j);
}
template <bool INV> __device__ __forceinline__ void fx_dft4(longlong2& a, longlong2& b, longlong2& c, longlong2& d) {
  const longlong2 t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = fx_rot<INV>(csub(b, d));
  a = cadd(t0, t2);
  c = csub(t0, t2);
  b = cadd(t1, t3);
  d = csub(t1, t3);
}
template <bool INV, int R> __device__ __forceinline__ void fx_dft(longlong2 (&v)[R]) {
  if constexpr (R == 2) {
    const longlong2 a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  } else if constexpr (R == 3) {
    fx_dft3<INV>(v[0], v[1], v[2]);
  } else if constexpr (R == 4) {
    fx_dft4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    fx_dft4<INV>(v[0], v[2], v[4], v[6]);
    fx_dft4<INV>(v[1], v[3], v[5], v[7]);
    // even outputs 0..3 in v[0], v[2], v[4], v[6], odd ones in v[1], v[3], v[5], v[7]
    const longlong2 o1 = fx_w8<INV>(v[3]), o2 = fx_rot<INV>(v[5]), o3 = fx_rot<INV>(fx_w8<INV>(v[7]));
    const longlong2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  } else if constexpr (R == 6) {
    // 6 = 2 x 3 by the prime-factor map: no twiddles
    longlong2 a0 = v[0], a1 = v[2], a2 = v[4], b0 = v[3], b1 = v[5], b2 = v[1];
    fx_dft3<INV>(a0, a1, a2);
    fx_dft3<INV>(b0, b1, b2);
    v[0] = cadd(a0, b0); v[3] = csub(a0, b0);
    v[4] = cadd(a1, b1); v[1] = csub(a1, b1);
    v[2] = cadd(a2, b2); v[5] = csub(a2, b2);
  } else {
    static_assert(R == 9, "radices 2, 3, 4, 6, 8, 9");
    // 3 x 3: x[3 a + b] -> X[k + 3 l], twiddles W9^{b k}
    fx_dft3<INV>(v[0], v[3], v[6]);
    fx_dft3<INV>(v[1], v[4], v[7]);
    fx_dft3<INV>(v[2], v[5], v[8]);
    auto w = [](longlong2 a, int k) {           // times W9 to the power 1, 2 or 4 (k = 0, 1, 2)
      const FxConst c = fx_const(fx_c9(k)), s = fx_const(fx_s9(k));
      return fx_cmul<!INV>(a, make_int4(c.h, c.l, s.h, s.l));
    };
    v[4] = w(v[4], 0);
    v[7] = w(v[7], 1);
    v[5] = w(v[5], 1);
    v[8] = w(v[8], 2);
    fx_dft3<INV>(v[0], v[1], v[2]);
    fx_dft3<INV>(v[3], v[4], v[5]);
    fx_dft3<INV>(v[6], v[7], v[8]);
    // v[3 k + l] holds X[k + 3 l]
    longlong2 t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
  }
}

// The e with 2^(e-1) <= v < 2^e, for a normal v > 0.
__device__ __forceinline__ int fx_bits_above(float v) { return (int)((__float_as_uint(v) >> 23) & 255) - 126; }

// High word of |x| (one less for exact negative powers of two).
__device__ __forceinline__ int fx_abs_hi(i64 x) { return (int)((u64)(x ^ (x >> 63)) >> 32); }

// One stage over G lines of length N that start at element `base`, by one warp.  Butterfly
// (block, j) takes the elements block R st + j + r st; its twiddles e^{-2 pi i j r / (R st)} are
// tw[(r - 1) st + j], so the lanes read consecutive entries.  UNIT (st = 1) has none: the last
// backward stage, which records the largest high words of the real and imaginary parts of each
// line in aux[2 line], aux[2 line + 1] if aux is given, and the first forward one, which scales
// line by 2^aux[line].  The first two stages (fine given, gs = 0 and 8) divide what they leave of line by
// 2^(byte of fine[fs line] at bit gs).
template <bool INV, int R, bool UNIT>
__device__ __forceinline__ void fx_stage(longlong2* buf, int base, int G, const FxPlan& pl, int s,
                                         const int4* __restrict__ tw, int* aux, const int* fine, int fs, int gs) {
  const int N = pl.N, nb = N / R, st = UNIT ? 1 : pl.stride[s];
  const FastDiv fb = pl.fnb[s], fst = pl.fst[s];
  const int lane = threadIdx.x & 31;
  const int total = G * nb;
  int mr = 0, mi = 0;
  for (int b = lane; b < total; b += 32) {
    const int line = G == 1 ? 0 : fb.div(b);
    const int jj = b - line * nb;
    const int blk = UNIT ? jj : fst.div(jj);
    const int j = UNIT ? 0 : jj - blk * st;
    const int i0 = base + line * N + blk * (R * st) + j;
    longlong2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = buf[fx_at(i0 + r * st)];
    if constexpr (!INV) {
      if constexpr (UNIT) {
        const int sh = aux[line];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = fx_shift2(v[r], sh);
      } else {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fx_cmul<false>(v[r], tw[(r - 1) * st + j]);
      }
    }
    fx_dft<INV, R>(v);
    if constexpr (INV && !UNIT) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = fx_cmul<true>(v[r], tw[(r - 1) * st + j]);
    }
    if constexpr (!(INV && UNIT)) {
      const int g = fine ? (fine[fs * line] >> gs) & 255 : 0;
      if (g) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[r].x = fx_down(v[r].x, g);
          v[r].y = fx_down(v[r].y, g);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) buf[fx_at(i0 + r * st)] = v[r];
    if constexpr (INV && UNIT) {
      if (aux) {
        int a = 0, c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) { a = max(a, fx_abs_hi(v[r].x)); c = max(c, fx_abs_hi(v[r].y)); }
        if (G == 1) { mr = max(mr, a); mi = max(mi, c); }
        else { atomicMax(&aux[2 * line], a); atomicMax(&aux[2 * line + 1], c); }
      }
    }
  }
  if constexpr (INV && UNIT) {
    if (aux && G == 1) {
      mr = __reduce_max_sync(0xffffffffu, mr);
      mi = __reduce_max_sync(0xffffffffu, mi);
      if (lane == 0) { aux[0] = mr; aux[1] = mi; }
    }
  }
  __syncwarp();
}

// The bits by which the scale of a line may lie above that of its L1 norm (exponent e) until the first
// stage, and the first two, are done, whose results are sums of only R and R R' values of at most
// `most` 2^e0: fx_fine_bits are given back as low byte after the first stage, second byte after the next.
__device__ __forceinline__ int fx_fine(const FxPlan& pl, bool inv, float most, int e0, int e) {
  if (pl.nst < 2 || !(most > 0.f) || e >= kFxZero) return 0;
  const int R = pl.radix[inv ? 0 : pl.nst - 1], R2 = R * pl.radix[inv ? 1 : pl.nst - 2];
  const int g = min(40, max(0, 61 - (e0 + fx_bits_above(most * (float)R * 1.001f)) - e));
  const int g2 = pl.nst < 3 ? 0 : min(g, max(0, 61 - (e0 + fx_bits_above(most * (float)R2 * 1.001f)) - e));
  return (g - g2) | g2 << 8;
}
__device__ __forceinline__ int fx_fine_bits(int f) { return (f & 255) + (f >> 8); }

// G lines of the plan's length by one warp (see fx_stage for aux and fine).
template <bool INV>
__device__ __forceinline__ void fx_fft(longlong2* buf, int base, int G, const FxPlan& pl, const int4* __restrict__ tw, int* aux,
                                       const int* fine, int fs) {
  for (int i = 0; i < pl.nst; ++i) {
    const int s = INV ? i : pl.nst - 1 - i;
    const int4* t = tw + pl.tw_off[s];
    const bool unit = s == pl.nst - 1;
    const int* f = i < 2 ? fine : nullptr;
#define MWF_FX(R_) case R_: if (unit) fx_stage<INV, R_, true>(buf, base, G, pl, s, t, aux, f, fs, 8 * i); else fx_stage<INV, R_, false>(buf, base, G, pl, s, t, aux, f, fs, 8 * i); break;
    switch (pl.radix[s]) {
      MWF_FX(8) MWF_FX(6) MWF_FX(4) MWF_FX(2) MWF_FX(3) MWF_FX(9)
      default: break;
    }
#undef MWF_FX
  }
}

// ---- products of the coupling: operands of at most 59 bits as h 2^30 + l, |l| <= 2^29 ----
struct FxLimbs { int h, l; };
struct FxAcc { i64 hi, cr; };      // hi 2^60 + cr 2^30
__device__ __forceinline__ FxLimbs fx_limbs(i64 x) {
  FxLimbs o;
  o.h = (int)((x + (1ll << 29)) >> 30);
  o.l = (int)((unsigned)(u64)x << 2) >> 2;
  return o;
}
// fx_limbs(fx_shift(x, sh)), the two roundings of the shifted value in one addition each
__device__ __forceinline__ FxLimbs fx_shift_limbs(i64 x, int sh) {
  const int up = sh > 0 ? sh : 0;
  const i64 t = fx_sar(fx_shl(x, up + 1), up - sh);
  FxLimbs o;
  o.h = (int)((t + ((1ll << 30) + 1)) >> 31);
  o.l = (int)(((unsigned)(u64)t + 1u) << 1) >> 2;
  return o;
}
__device__ __forceinline__ FxLimbs fx_twice(FxLimbs a) { return FxLimbs{2 * a.h, 2 * a.l}; }
// k = 1 ... 5 times an operand of 58 bits (5 l would overflow)
__device__ __forceinline__ FxLimbs fx_times(FxLimbs a, int k) {
  return k <= 4 ? FxLimbs{k * a.h, k * a.l} : fx_limbs(k * (((i64)a.h << 30) + a.l));
}
// For operands of 58 and 59 bits (58 and 58 in the y direction) and the largest weights of a coupling row, 12
// (x, z) and 24 (y, the factors of fx_times included), hi stays below 2^61 and cr below 2^63; the products of two low
// limbs (at most 2^-59 of the largest product) are dropped.
__device__ __forceinline__ void fx_mac(FxAcc& a, FxLimbs v, FxLimbs d) {
  a.hi = fx_madw(v.h, d.h, a.hi);
  a.cr = fx_madw(v.h, d.l, fx_madw(v.l, d.h, a.cr));
}
__device__ __forceinline__ void fx_msb(FxAcc& a, FxLimbs v, FxLimbs d) { fx_mac(a, FxLimbs{-v.h, -v.l}, d); }
// The sum times 2^(left - 60), rounded; 0 <= left <= 29, |.| < 2^63.
__device__ __forceinline__ i64 fx_sum(FxAcc a, int left) {
  return fx_shl(a.hi, left) + fx_sar(a.cr + fx_shl(1, 29 - left), 30 - left);
}

}  // namespace mwf
