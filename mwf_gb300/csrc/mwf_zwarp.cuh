// FP32 z pass of the line lengths that have no compile-time plan (sm_103a): in-place transforms, a
// warp per line, any NN = 2^a 3^b.
//
// The work item is (run, first x line x0): L x lines and all three z-subsets z = s + 3q of them, as
// in the batched pass (mwf_zbatch.cuh), whose arithmetic it follows: packed pairs of u, v, w and
// (d/dx f, d/dz f) pairs backward, the coupling per point in registers (udotgradu, modes.M4.f90:14-28
// / modes.M6.f90:14-20), the products forward, the subsets summed.  The transforms are decimation
// in frequency backward and in time forward, in place (mwf_fx.cuh has the same scheme): a warp
// fills, transforms and later splits its own lines with warp barriers alone, no second buffer is
// needed and the order of the points in between does not matter, so the CTA synchronises twice per
// item.  Where a CTA holds one long line of each field a team of two warps takes a line.
// z_nonlinear_kernel, which these runs took before, runs 16 tasks per subset with a dozen
// CTA barriers each.  NS = 3 holds the three subsets' lines at once; where they do not fit a CTA,
// NS = 1 goes through the subsets in turn and adds their outputs in NLT.
#pragma once
#include "mwf_kernels.cuh"
#include "nl_gen.cuh"

namespace mwf {

// Place of element i of a line.  With one pad element after every (even) group of the last stage the
// strided butterflies spread over the banks, and the elements of a butterfly are equally spaced in every
// stage (the stage strides are multiples of the last radix), so an element costs one addition.
__device__ __forceinline__ int zw_at(const FxPlan& pl, int i) { return i + pl.fpad.div(i); }

template <bool INV> __device__ __forceinline__ void zw_dft6(float2* v) {
  // 6 = 2 x 3 by the prime-factor map: no twiddles
  float2 a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
  dft3<float>(a, INV);
  dft3<float>(b, INV);
  v[0] = cadd(a[0], b[0]); v[3] = csub(a[0], b[0]);
  v[4] = cadd(a[1], b[1]); v[1] = csub(a[1], b[1]);
  v[2] = cadd(a[2], b[2]); v[5] = csub(a[2], b[2]);
}
template <bool INV> __device__ __forceinline__ void zw_dft9(float2* v) {
  float2 y[3][3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    float2 t[3] = {v[b], v[b + 3], v[b + 6]};
    dft3<float>(t, INV);
#pragma unroll
    for (int k = 0; k < 3; ++k) y[b][k] = t[k];
  }
  y[1][1] = wmul<float>(y[1][1], 0.76604444311897803520f, 0.64278760968653932632f, INV);
  y[1][2] = wmul<float>(y[1][2], 0.17364817766693034885f, 0.98480775301220805937f, INV);
  y[2][1] = wmul<float>(y[2][1], 0.17364817766693034885f, 0.98480775301220805937f, INV);
  y[2][2] = wmul<float>(y[2][2], -0.93969262078590838405f, 0.34202014332566873304f, INV);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float2 t[3] = {y[0][k], y[1][k], y[2][k]};
    dft3<float>(t, INV);
#pragma unroll
    for (int l = 0; l < 3; ++l) v[k + 3 * l] = t[l];
  }
}
template <bool INV, int R> __device__ __forceinline__ void zw_dft(float2* v) {
  if constexpr (R == 6) zw_dft6<INV>(v);
  else if constexpr (R == 9) zw_dft9<INV>(v);
  else dftR<float, R>(v, INV);
}

// Synchronise the TW warps of a team (one warp, or the two of an aligned pair).
template <int TW> __device__ __forceinline__ void zw_sync() {
  if constexpr (TW == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + (int)(threadIdx.x / (32 * TW))), "n"(32 * TW) : "memory");
}
// One stage of `lines` lines of the plan's length from element `base`, by a team (see fx_stage).
template <bool INV, int R, int TW>
__device__ __forceinline__ void zw_stage(float2* buf, int base, int lines, const FxPlan& pl, int s, const float2* tw) {
  const int nb = pl.N / R, st = pl.stride[s], step = pl.step[s], bstep = pl.bstep[s], LS = pl.LS;
  const FastDiv fb = pl.fnb[s], fst = pl.fst[s];
  for (int b = threadIdx.x & (32 * TW - 1); b < lines * nb; b += 32 * TW) {
    const int line = fb.div(b);
    const int jj = b - line * nb;
    const int blk = fst.div(jj);
    const int j = jj - blk * st;
    float2* const at = buf + (base + line * LS + blk * bstep + zw_at(pl, j));
    const float2* const w = tw + j - st;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = at[r * step];
    if (!INV && st > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r * st]);
    }
    zw_dft<INV, R>(v);
    if (INV && st > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmulc(v[r], w[r * st]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) at[r * step] = v[r];
  }
  zw_sync<TW>();
}
template <bool INV, int TW>
__device__ __forceinline__ void zw_fft(float2* buf, int base, int lines, const FxPlan& pl, const float2* tw) {
  for (int i = 0; i < pl.nst; ++i) {
    const int s = INV ? i : pl.nst - 1 - i;
    const float2* t = tw + pl.tw_off[s];
    switch (pl.radix[s]) {
      case 2: zw_stage<INV, 2, TW>(buf, base, lines, pl, s, t); break;
      case 3: zw_stage<INV, 3, TW>(buf, base, lines, pl, s, t); break;
      case 4: zw_stage<INV, 4, TW>(buf, base, lines, pl, s, t); break;
      case 6: zw_stage<INV, 6, TW>(buf, base, lines, pl, s, t); break;
      case 8: zw_stage<INV, 8, TW>(buf, base, lines, pl, s, t); break;
      case 9: zw_stage<INV, 9, TW>(buf, base, lines, pl, s, t); break;
      case 12: zw_stage<INV, 12, TW>(buf, base, lines, pl, s, t); break;
      case 16: zw_stage<INV, 16, TW>(buf, base, lines, pl, s, t); break;
      default: break;
    }
  }
}

template <int K0, int NS, int NT, int MINB, int TW>
__global__ void __launch_bounds__(NT, MINB) z_warp_kernel(const RunDesc* __restrict__ runs, const WorkItem* __restrict__ items) {
  constexpr int KK = 3 * K0 - 1, NPAIR = (KK + 1) / 2, NTR = NPAIR + KK;
  constexpr int LN = 32 * TW, NW = NT / LN;           // threads of a team, teams
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const WorkItem wi = items[blockIdx.x];
  const RunDesc& R = runs[wi.run];
  if (!R.active) return;
  const int X = R.X, Q = R.NN, x0 = wi.a;
  const int L = min(R.zw_lines, X - x0);
  const FxPlan& pl = R.zw_plan;
  const int LS = pl.LS, TS = NS * L * LS;             // line (t, l, s) at t TS + (l NS + s) LS
  float2* buf = reinterpret_cast<float2*>(smem_raw);
  float2* tw = buf + (size_t)NTR * TS;                // [Q] stage twiddles
  const int team = threadIdx.x / LN, lane = threadIdx.x % LN;
  const float2* __restrict__ T = reinterpret_cast<const float2*>(R.T) + (size_t)x0 * Q;
  float2* __restrict__ NLT = reinterpret_cast<float2*>(R.NLT) + (size_t)x0 * Q;
  const size_t fstride = (size_t)X * Q;
  const float2* __restrict__ om = reinterpret_cast<const float2*>(R.twZ);     // e^{-2 pi i t/Z}
  const float gam = R.gamma_f;
  const float hscale = (float)(0.5 * R.scale);        // 1/2 of the Hermitian split times 1/(XZ)
  for (int i = threadIdx.x; i < Q; i += NT) tw[i] = R.zw_tw[i];
  const int G = max(1, min(L, 128 / Q));              // x lines of a warp's task
  const int groups = (L + G - 1) / G;
  // slot n < (Q+1)/2 of a line is the pair (n, Q-n); slot 0 is n = 0 with, for even Q, n = Q/2
  const int slots = (Q + 1) / 2;
  const bool even = (Q & 1) == 0;
  const FastDiv fSl = make_fastdiv(slots);
  __syncthreads();

#pragma unroll 1
  for (int s0 = 0; s0 < 3; s0 += NS) {
    // ---- fill and backward transforms; a team's next rows are loaded while it transforms ----
    struct Task { const float2 *pa, *pb; int t, l0, nl, total; bool der, two; };
    struct In { float2 Pa, Ra, Pb, Rb; };
    auto task = [&](int i) {
      Task k;
      k.t = i / groups;
      k.l0 = (i - k.t * groups) * G;
      k.nl = min(G, L - k.l0);
      k.total = i < NTR * groups ? k.nl * slots : 0;
      k.der = k.t >= NPAIR;
      k.two = k.der || 2 * k.t + 1 < KK;
      const int fa = k.der ? KK + k.t - NPAIR : 2 * k.t, fb = k.der ? k.t - NPAIR : (k.two ? 2 * k.t + 1 : fa);
      k.pa = T + (size_t)fa * fstride + (size_t)k.l0 * Q;
      k.pb = T + (size_t)fb * fstride + (size_t)k.l0 * Q;
      return k;
    };
    auto load = [&](const Task& k, int idx) {
      const int l = fSl.div(idx), sl = idx - l * slots;
      const int n = l * Q + (sl ? sl : (even ? Q / 2 : 0)), nq = l * Q + (sl ? Q - sl : 0);
      In v;
      v.Pa = k.pa[n]; v.Ra = k.pa[nq]; v.Pb = k.pb[n]; v.Rb = k.pb[nq];
      return v;
    };
    Task nt = task(team);
    In nx;
    if (lane < nt.total) nx = load(nt, lane);
    for (int i = team; i < NTR * groups; i += NW) {
      const Task ct = nt;
      const int t = ct.t, l0 = ct.l0, nl = ct.nl, total = ct.total;
      const bool der = ct.der, two = ct.two;
      for (int idx = lane; idx < total; idx += LN) {
        const float2 Pa = nx.Pa;
        float2 Ra = nx.Ra, Pb = nx.Pb, Rb = nx.Rb;
        if (idx + LN < total) nx = load(ct, idx + LN);
        if (!two) Pb = Rb = make_float2(0.f, 0.f);
        const int l = fSl.div(idx), sl = idx - l * slots;
        const int n = sl ? sl : (even ? Q / 2 : 0), nq = sl ? Q - sl : n;
        const int base = t * TS + (l0 + l) * NS * LS;
        const int an = base + zw_at(pl, n), aq = base + zw_at(pl, nq);
        if (sl == 0) {                                // H = Re X_0; the z derivative has none
          const float2 h = make_float2(Ra.x, der ? 0.f : Rb.x);
#pragma unroll
          for (int k = 0; k < NS; ++k) buf[base + k * LS] = h;
          Ra = Pa;
          Rb = Pb;
        }
        // packed lines at n and Q-n: H[n] = w U + (eps w) V and H[Q-n] = conj(eps w) U' + conj(w) V'
        // (see z_nonlinear_kernel)
        float2 U, V, U2, V2;
        if (der) {
          const float gn = gam * (float)n, gq = gam * (float)nq;
          U = make_float2(fmaf(-gn, Pb.x, Pa.x), fmaf(-gn, Pb.y, Pa.y));
          V = make_float2(fmaf(gq, Rb.x, Ra.x), -fmaf(gq, Rb.y, Ra.y));
          U2 = make_float2(fmaf(-gq, Rb.x, Ra.x), fmaf(-gq, Rb.y, Ra.y));
          V2 = make_float2(fmaf(gn, Pb.x, Pa.x), -fmaf(gn, Pb.y, Pa.y));
        } else {
          U = make_float2(Pa.x - Pb.y, Pa.y + Pb.x);
          V = make_float2(Ra.x + Rb.y, Rb.x - Ra.y);
          U2 = make_float2(Ra.x - Rb.y, Ra.y + Rb.x);
          V2 = make_float2(Pa.x + Pb.y, Pb.x - Pa.y);
        }
#pragma unroll
        for (int k = 0; k < NS; ++k) {
          const int s = s0 + k;
          float2 Hn, Hq;
          if (s == 0) {
            Hn = cadd(U, V);
            Hq = cadd(U2, V2);
          } else {
            const float2 tz = __ldg(&om[n * s]), tq = __ldg(&om[nq * s]);     // conj(w), eps w
            Hn = cmac(cmulc(U, tz), V, tq);
            Hq = cmac(cmulc(U2, tq), V2, tz);
          }
          if (sl || even) buf[an + k * LS] = Hn;
          if (sl) buf[aq + k * LS] = Hq;
        }
      }
      nt = task(i + NW);
      if (lane < nt.total) nx = load(nt, lane);
      zw_sync<TW>();
      zw_fft<true, TW>(buf, t * TS + l0 * NS * LS, nl * NS, pl, tw);
    }
    __syncthreads();

    // ---- coupling ----
    const FastDiv fQ = make_fastdiv(Q);
    for (int e = threadIdx.x; e < NS * L * Q; e += NT) {
      const int line = fQ.div(e);
      float2* const at = buf + line * LS + zw_at(pl, e - line * Q);
      float pv[KK], nl[KK];
#pragma unroll
      for (int t = 0; t < NPAIR; ++t) {
        const float2 v = at[t * TS];
        pv[2 * t] = v.x;
        if (2 * t + 1 < KK) pv[2 * t + 1] = v.y;
      }
      if constexpr (K0 == 4) nl_y_4<float>(pv, nl); else nl_y_6<float>(pv, nl);
#pragma unroll
      for (int J = 0; J < KK; ++J) {
        const float2 v = at[(NPAIR + J) * TS];
        nl_xz_rt<K0, float>(J, pv, v.x, v.y, nl);
      }
#pragma unroll
      for (int t = 0; t < NPAIR; ++t) at[t * TS] = make_float2(nl[2 * t], 2 * t + 1 < KK ? nl[2 * t + 1] : 0.f);
    }
    __syncthreads();

    // ---- forward transforms, split, sum over the subsets, store ----
    for (int i = team; i < NPAIR * groups; i += NW) {
      const int t = i / groups, l0 = (i - t * groups) * G, nl = min(G, L - l0);
      const int first = t * TS + l0 * NS * LS;
      zw_fft<false, TW>(buf, first, nl * NS, pl, tw);
      const bool two = 2 * t + 1 < KK;
      float2* __restrict__ oa = NLT + (size_t)(2 * t) * fstride + (size_t)l0 * Q;
      float2* __restrict__ ob = oa + fstride;
      auto put = [&](int o, float2 a, float2 b) {
        oa[o] = a;
        if (two) ob[o] = b;
      };
      const float2 none = make_float2(0.f, 0.f);
      for (int idx = lane; idx < nl * slots; idx += LN) {
        const int l = fSl.div(idx), sl = idx - l * slots;
        const int base = first + l * NS * LS, o = l * Q;
        const int n = sl ? sl : (even ? Q / 2 : 0), nq = sl ? Q - sl : n;
        const int an = base + zw_at(pl, n), aq = base + zw_at(pl, nq);
        const int on = o + n, oq = o + (sl ? nq : 0);
        const bool hasn = sl || even;
        // sums over the subsets, with the subset's factor fused; one after the other: on top of this thread's sums of
        // the earlier ones
        float2 An = none, Bn = none, Aq = none, Bq = none;
        if (NS == 1 && s0 > 0) {
          if (hasn) { An = oa[on]; if (two) Bn = ob[on]; }
          Aq = oa[oq];
          if (two) Bq = ob[oq];
        }
#pragma unroll
        for (int k = 0; k < NS; ++k) {
          const int s = s0 + k;
          const float2 g = buf[an + k * LS], m = buf[aq + k * LS];
          const float2 A = make_float2(hscale * (g.x + m.x), hscale * (g.y - m.y));
          const float2 B = make_float2(hscale * (g.y + m.y), hscale * (m.x - g.x));
          if (s == 0) {
            An = A;
            Bn = B;
          } else {
            const float2 tz = __ldg(&om[n * s]);
            An = cmac(An, A, tz);
            Bn = cmac(Bn, B, tz);
          }
          if (sl == 0) {                              // n = 0
            const float2 z = buf[base + k * LS];
            Aq.x = __fmaf_rn(2.f * hscale, z.x, Aq.x);
            Bq.x = __fmaf_rn(2.f * hscale, z.y, Bq.x);
          } else if (s == 0) {
            Aq = cconj(A);
            Bq = cconj(B);
          } else {
            const float2 tq = __ldg(&om[nq * s]);
            Aq = cmac(Aq, cconj(A), tq);
            Bq = cmac(Bq, cconj(B), tq);
          }
        }
        if (hasn) put(on, An, Bn);
        put(oq, Aq, Bq);
      }
    }
    if (NS == 1) __syncthreads();                     // the next subset's fill takes the lines
  }
}

}  // namespace mwf
