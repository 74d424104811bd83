// FP32 x passes of the lengths that have no compile-time plan (sm_103a): the arithmetic of
// mwf_xbatch.cuh -- three interleaved subsets x = s + 3q of length MM per line -- with the in-place
// transforms of mwf_zwarp.cuh, a warp per subset line, any MM = 2^a 3^b.
//
// x forward: item (run, first column n0, wall-normal mode k): u_k, v_k (k >= 1), w_k and their x
//   derivatives (var_mpt2spec + vel_addlam + var_spec_grad, variables.f90:390-434,600-612,
//   velocity.f90:76-82) of nb columns, xw_nd of {field, derivative} at a time
// x inverse: item (run, n0, k): the three fields forward, var_spec2mpt (variables.f90:440-480) and
//   the update of vel_TS (velocity.f90:21-41) as in xi_batched_body
// Consecutive threads take consecutive columns of T and NLT (nb a power of two: 32-byte sectors from
// nb = 4 on), and the line transforms need warp barriers alone.  The kernels these runs took before
// transform lines of 3MM points in three or four CTA-wide stages of run-time radix.
#pragma once
#include "mwf_zwarp.cuh"

namespace mwf {

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) x_forward_warp_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, MM = R.MM, NN = R.NN, KK = R.KK, M = R.M, K = R.K, K0 = R.K0;
  const int n0 = wi.a, k = wi.b, nbw = R.xw_fnb, nd = R.xw_nd;
  const int nb = min(nbw, NN - n0);
  const FxPlan& pl = R.xw_plan;
  const int LS = pl.LS;
  float2* buf = reinterpret_cast<float2*>(smem_raw);  // line (d, l, s) at ((d nb + l) 3 + s) LS
  float2* tw = buf + 3 * nd * nbw * LS;
  for (int i = threadIdx.x; i < MM; i += NT) tw[i] = R.xw_tw[i];
  const int warp = threadIdx.x >> 5;
  constexpr int NW = NT / 32;
  const float2* __restrict__ c = reinterpret_cast<const float2*>(R.c);
  const float2* __restrict__ twX = reinterpret_cast<const float2*>(R.twX);
  float2* __restrict__ T = reinterpret_cast<float2*>(R.T);
  const FastDiv fMM = make_fastdiv(MM);
  const float k1 = kbeta<float>(k), alpha = R.alpha_f, gamma = R.gamma_f;
  const int lw = 31 - __clz(nbw);
  const int lines = 3 * nb * nd, G = max(1, min(lines, 256 / MM));
  for (int pass = 0; pass < (k >= 1 ? 3 : 2) * 2 / nd; ++pass) {
    const int ci = nd == 2 ? pass : pass >> 1, d0 = nd == 2 ? 0 : pass & 1;
    const int comp = (k == 0 && ci == 1) ? 2 : ci;    // v_0 does not exist
    const int fs = comp == 0 ? k : (comp == 1 ? K0 - 1 + k : 2 * K0 - 1 + k);
    const size_t ra = (size_t)(comp == 1 ? k + K0 - 1 : k) * M, rb = (size_t)(k + K0 - 1) * M;
    const bool hasb = comp != 1 && k >= 1;
    // fill: a = value at m = j, b = value at m = j - MM; subset s has the spectrum
    // e^{2 pi i js/X} (a + e^{-2 pi i s/3} b)
    for (int e = threadIdx.x; e < nb * MM; e += NT) {
      const int l = fMM.div(e);
      const int j = e - l * MM, n = n0 + l;
      const float2* __restrict__ col = c + (size_t)n * K * M;
      const float n1 = gamma * (float)n;
      const int msn = j == 0 ? 0 : j + M - MM;        // slot of m = j - MM
      const float2 zero = make_float2(0.f, 0.f);
      const float2 Aj = col[ra + j], An = col[ra + msn];
      const float2 Bj = hasb ? col[rb + j] : zero, Bn = hasb ? col[rb + msn] : zero;
      auto field = [&](float2 a, float2 b, float m1) {
        if (comp == 1) {
          const float H = fmaf(-m1, m1, -(n1 * n1));
          return make_float2(-a.x * H, -a.y * H);
        }
        if (comp == 0) return make_float2(-fmaf(-a.y, n1, b.y * k1 * m1), fmaf(-a.x, n1, b.x * k1 * m1));
        return make_float2(-fmaf(a.y, m1, b.y * k1 * n1), fmaf(a.x, m1, b.x * k1 * n1));
      };
      const float mp = alpha * (float)j, mn = alpha * (float)(j - MM);
      float2 v = field(Aj, Bj, mp), w = field(An, Bn, mn);
      if (j == 0) {
        w = zero;
        if (n == 0) {                                 // mean flows: u_k = psi_k, w_k = phi_k (k >= 1)
          v = zero;
          if (comp == 0 && k >= 1) v = Aj;
          if (comp == 2 && k >= 1) v = Bj;
          if (k == 1 && comp == 0) v.x += (float)R.cth;
          if (k == 1 && comp == 2) v.x += (float)R.sth;
        }
      }
      const float2 t1 = twX[j], t2 = twX[2 * j];
      for (int i = 0; i < nd; ++i) {
        float2 a = v, b = w;
        if (d0 + i) {
          a = make_float2(-v.y * mp, v.x * mp);
          b = make_float2(-w.y * mn, w.x * mn);
        }
        float2* const at = buf + (i * nb + l) * 3 * LS + zw_at(pl, j);
        const float r3 = 0.86602540378443864676f;
        const float hx = fmaf(-0.5f, b.x, a.x), hy = fmaf(-0.5f, b.y, a.y);
        at[0] = cadd(a, b);
        at[LS] = cmulc(make_float2(fmaf(r3, b.y, hx), fmaf(-r3, b.x, hy)), t1);
        at[2 * LS] = cmulc(make_float2(fmaf(-r3, b.y, hx), fmaf(r3, b.x, hy)), t2);
      }
    }
    __syncthreads();
    for (int t = warp * G; t < lines; t += NW * G) zw_fft<true, 1>(buf, t * LS, min(G, lines - t), pl, tw);
    __syncthreads();
    for (int e = threadIdx.x; e < (X << lw); e += NT) {
      const int l = e & (nbw - 1), sp = e >> lw;      // s MM + position
      if (l >= nb) continue;
      const int s = fMM.div(sp), p = sp - s * MM;
      const int x = s + 3 * R.xw_rev[p];
      for (int i = 0; i < nd; ++i)
        T[((size_t)((d0 + i) * KK + fs) * X + x) * NN + n0 + l] = buf[((i * nb + l) * 3 + s) * LS + zw_at(pl, p)];
    }
    __syncthreads();
  }
}

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) x_inverse_warp_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, MM = R.MM, NN = R.NN, M = R.M, K0 = R.K0, K = R.K;
  const int n0 = wi.a, k = wi.b, nbw = R.xw_inb;
  const int nb = min(nbw, NN - n0);
  const FxPlan& pl = R.xw_plan;
  const int LS = pl.LS;
  float2* buf = reinterpret_cast<float2*>(smem_raw);  // line (comp, l, s) at ((comp nb + l) 3 + s) LS
  float2* tw = buf + 9 * nbw * LS;
  for (int i = threadIdx.x; i < MM; i += NT) tw[i] = R.xw_tw[i];
  const float2* __restrict__ NLT = reinterpret_cast<const float2*>(R.NLT);
  const size_t fstride = (size_t)X * NN;
  const FastDiv fMM = make_fastdiv(MM), fX = make_fastdiv(X);
  const int lw = 31 - __clz(nbw);
  {
    const int l = threadIdx.x & (nbw - 1);
    if (l < nb) {
#pragma unroll 4
      for (int r = threadIdx.x >> lw; r < 3 * X; r += NT >> lw) {
        const int comp = fX.div(r), sp = r - comp * X;
        const int s = fMM.div(sp), p = sp - s * MM;
        const int f = comp == 0 ? k : comp == 1 ? K0 + k - 1 : 2 * K0 - 1 + k;
        float2 v = make_float2(0.f, 0.f);
        if (!(comp == 1 && k == 0)) v = NLT[(size_t)f * fstride + (size_t)(s + 3 * R.xw_rev[p]) * NN + n0 + l];
        buf[((comp * nb + l) * 3 + s) * LS + zw_at(pl, p)] = v;
      }
    }
  }
  __syncthreads();
  {
    const int lines = 9 * nb, G = max(1, min(lines, 256 / MM));
    for (int t = (threadIdx.x >> 5) * G; t < lines; t += NT / 32 * G) zw_fft<false, 1>(buf, t * LS, min(G, lines - t), pl, tw);
  }
  __syncthreads();

  // combine the subsets, var_spec2mpt and the update (see xi_batched_body)
  float2* __restrict__ c = reinterpret_cast<float2*>(R.c);
  float2* __restrict__ onl = reinterpret_cast<float2*>(R.onl);
  const float2* __restrict__ twX = reinterpret_cast<const float2*>(R.twX);
  const size_t csz = (size_t)NN * K * M;
  const float* __restrict__ a_hi = reinterpret_cast<const float*>(R.inv_lhs);
  const float* __restrict__ a_lo = a_hi + csz;
  const float* __restrict__ bnl = reinterpret_cast<const float*>(R.rhs);
  const bool first = *R.nst != 0;
  const float kb1 = kbeta<float>(k), alpha = R.alpha_f, gamma = R.gamma_f;
  const FastDiv fM = make_fastdiv(M);
  for (int o = threadIdx.x; o < nb * M; o += NT) {
    const int l = fM.div(o);
    const int ms = o - l * M, n = n0 + l;
    const size_t i0 = ((size_t)n * K + k) * M + ms, i1 = i0 + (size_t)(K0 - 1) * M;
    const float2 c0 = c[i0], o0 = onl[i0];
    const float ah0 = a_hi[i0], al0 = a_lo[i0], b0 = bnl[i0];
    float2 c1 = make_float2(0.f, 0.f), o1 = c1;
    float ah1 = 0.f, al1 = 0.f, b1 = 0.f;
    if (k > 0) {
      c1 = c[i1]; o1 = onl[i1];
      ah1 = a_hi[i1]; al1 = a_lo[i1]; b1 = bnl[i1];
    }
    const int m = signed_m(ms, MM, M);
    const int j = m >= 0 ? m : m + MM;
    const float2 w1 = twX[m >= 0 ? m : m + X], w2 = twX[m >= 0 ? 2 * m : 2 * m + X];
    const float2* const at = buf + l * 3 * LS + zw_at(pl, j);
    float2 sp[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float2* const q = at + i * nb * 3 * LS;
      sp[i] = cadd(cadd(q[0], cmul(q[LS], w1)), cmul(q[2 * LS], w2));
    }
    const float2 su = sp[0], sv = sp[1], sw = sp[2];
    const float m1 = alpha * (float)m, n1 = gamma * (float)n;
    const float H = fmaf(-m1, m1, -(n1 * n1));
    float2 nphi, npsi;
    nphi.x = fmaf(sv.x, H, -(su.y * m1 * kb1 + sw.y * n1 * kb1));
    nphi.y = fmaf(sv.y, H, su.x * m1 * kb1 + sw.x * n1 * kb1);
    npsi.x = fmaf(sw.y, m1, -(su.y * n1));
    npsi.y = -fmaf(sw.x, m1, -(su.x * n1));
    if (ms == 0 && n == 0) {
      if (k == 0) npsi = make_float2(0.f, 0.f);
      else {
        npsi = make_float2(-su.x, -su.y);
        nphi = make_float2(-sw.x, -sw.y);
      }
    }
    auto update = [](float ah, float al, float b, float cv, float nv, float onv) {
      const float ph = __fmul_rn(ah, cv);             // not contracted: ph + pl = ah*cv exactly
      const float pl_ = fmaf(ah, cv, -ph);
      return __fadd_rn(ph, fmaf(b, fmaf(3.f, nv, -onv), fmaf(al, cv, pl_)));
    };
    {
      const float2 ov = first ? npsi : o0;
      float x = update(ah0, al0, b0, c0.x, npsi.x, ov.x);
      const float y = update(ah0, al0, b0, c0.y, npsi.y, ov.y);
      if (k == 0 && ms == 0 && n == 0) x = 0.f;
      c[i0] = make_float2(x, y);
      onl[i0] = npsi;
    }
    if (k > 0) {
      const float2 ov = first ? nphi : o1;
      c[i1] = make_float2(update(ah1, al1, b1, c1.x, nphi.x, ov.x), update(ah1, al1, b1, c1.y, nphi.y, ov.y));
      onl[i1] = nphi;
    }
  }
}

}  // namespace mwf
