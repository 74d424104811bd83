// C-ABI implementation (include/mwf_gpu.h): plans, FP64 tables, device arena, work lists,
// CUDA-graph replay of the timestep, state copies and the energy diagnostic.
#include <cuda.h>
#include <cmath>
#include <cstddef>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <map>
#include <vector>
#include <algorithm>

#include "../../include/mwf_gpu.h"
#include "mwf_common.cuh"
#include "mwf_launch.h"

using namespace mwf;

namespace {

thread_local char g_err[512];

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

#define CK(call)                                                                          \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess) return fail(MWF_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

constexpr int kMaxLen = 4096;      // longest x line (3*MM) supported by the plans
constexpr int kMaxNN = 1024;       // longest z half-line (NN) supported by the z pass
constexpr size_t kSmemLimit = 200 * 1024;

bool is_23_smooth(int n) {
  if (n < 1) return false;
  while (n % 2 == 0) n /= 2;
  while (n % 3 == 0) n /= 3;
  return n == 1;
}

// Radix plan for N = 2^a 3^b with radices up to maxr (8, 12 or 16): as few stages as
// possible.  Each 3 pairs with a 4 into a radix-12 stage while both are left (maxr >= 12),
// leftover 3s are radix-3 stages, and the power of two is split into the fewest stages of
// 16/8/4/2, balanced toward 8s.
bool make_plan(int N, FftPlanDev& pl, int maxr) {
  if (!is_23_smooth(N) || N < 2) return false;
  int a = 0, b = 0, rest = N;
  while (rest % 2 == 0) { rest /= 2; ++a; }
  while (rest % 3 == 0) { rest /= 3; ++b; }
  std::vector<int> rad;
  if (maxr >= 12) {
    while (b > 0 && a >= 2) { rad.push_back(12); --b; a -= 2; }
  }
  while (b > 0) { rad.push_back(3); --b; }
  static const int p16[13][3] = {{0, 0, 0}, {2, 0, 0}, {4, 0, 0}, {8, 0, 0}, {16, 0, 0}, {8, 4, 0},
                                 {8, 8, 0}, {16, 8, 0}, {16, 16, 0}, {8, 8, 8}, {16, 8, 8}, {16, 16, 8},
                                 {16, 16, 16}};
  while (a > 0) {
    if (maxr >= 16) {
      const int take = std::min(a, 12);
      for (int i = 0; i < 3 && p16[take][i]; ++i) rad.push_back(p16[take][i]);
      a -= take;
    } else {
      const int take = a >= 3 ? 3 : a;
      rad.push_back(1 << take);
      a -= take;
    }
  }
  if ((int)rad.size() > MWF_MAX_STAGES) return false;
  pl.N = N;
  pl.nst = 0;
  int ns = 1;
  for (int r : rad) {
    pl.radix[pl.nst] = r;
    pl.ns[pl.nst] = ns;
    pl.fnb[pl.nst] = make_fastdiv(N / r);
    pl.fns[pl.nst] = make_fastdiv(ns);
    ++pl.nst;
    ns *= r;
  }
  return ns == N;
}

// cos and sin of 2 pi t / N in long double, the argument folded into [0, pi/4]: with 4t = q N + r the
// angle is (q + r/N) quarter turns, and r > N/2 swaps the two.  first(r), r <= N/2, gives them for
// r/N of a quarter turn.
template <typename F>
void unit_root(int N, int t, F&& first, long double& c, long double& s) {
  const int q = (int)(4LL * t / N), r = (int)(4LL * t - (long long)q * N);
  long double a, b;                            // cos, sin of r/N quarter turns
  if (2 * r <= N) first(r, a, b);
  else first(N - r, b, a);
  switch (q & 3) {
    case 0: c = a; s = b; break;
    case 1: c = -b; s = a; break;
    case 2: c = -a; s = -b; break;
    default: c = b; s = -a; break;
  }
}
void first_octant(int N, int r, long double& c, long double& s) {
  const long double h = 0.707106781186547524400844362104849039L, quarter = 1.570796326794896619231321691639751442L;
  if (r == 0) { c = 1.0L; s = 0.0L; return; }
  if (2 * r == N) { c = s = h; return; }
  const long double a = quarter * (long double)r / (long double)N;
  c = cosl(a);
  s = sinl(a);
}

// tw[t] = exp(-2 pi i t / N) for t in [t0, t0 + cnt), evaluated in long double and rounded
// once; out receives 2*cnt values (re, im interleaved).
template <typename T>
void twiddles_into(int N, int t0, int cnt, T* out) {
  for (int t = t0; t < t0 + cnt; ++t) {
    long double c, s;
    unit_root(N, t, [&](int r, long double& a, long double& b) { first_octant(N, r, a, b); }, c, s);
    out[2 * (size_t)(t - t0)] = (T)c;
    out[2 * (size_t)(t - t0) + 1] = (T)(-s);
  }
}

// The whole table in long double; each first-octant value is evaluated once (N/8 of them where
// 4 divides N: long double functions take 0.7 us on the Grace host).
std::vector<long double> twiddles(int N) {
  std::vector<long double> out(2 * (size_t)N), oct(2 * ((size_t)N / 2 + 1));
  std::vector<char> have((size_t)N / 2 + 1, 0);
  auto first = [&](int r, long double& a, long double& b) {
    if (!have[r]) {
      first_octant(N, r, oct[2 * (size_t)r], oct[2 * (size_t)r + 1]);
      have[r] = 1;
    }
    a = oct[2 * (size_t)r];
    b = oct[2 * (size_t)r + 1];
  };
  for (int t = 0; t < N; ++t) {
    long double c, s;
    unit_root(N, t, first, c, s);
    out[2 * (size_t)t] = c;
    out[2 * (size_t)t + 1] = -s;
  }
  return out;
}

// A twiddle (re, im) times 2^62 as two 32-bit limbs per part (FxConst: high, signed low), the low
// limbs kept off -2^31 so that they can be negated.
int4 fx_twiddle(const long double* v) {
  int out[4];
  for (int i = 0; i < 2; ++i) {
    long long w = llroundl(v[i] * 4611686018427387904.0L);
    if ((unsigned)w == 0x80000000u) ++w;
    const int l = (int)(unsigned)w;
    out[2 * i] = (int)((w - l) >> 32);
    out[2 * i + 1] = l;
  }
  return make_int4(out[0], out[1], out[2], out[3]);
}

// Radices of the in-place transforms of length N: the fewest stages, with radices up to 9 in fixed
// point (a butterfly of 12 or 16 would not leave 128 registers a thread) and up to 16 in FP32.
std::vector<int> inplace_radices(int N, bool fx) {
  static const int all[] = {16, 12, 9, 8, 6, 4, 3, 2};
  std::vector<int> cur, best;
  int best_sum = 0;
  // depth-first over non-increasing radices: fewest stages, then (FP32, from 512 on) the fewest of radix 9, whose
  // inner twiddles round most of its outputs once more, then (FP32) the least padding (the last radix, below),
  // then the smallest sum.  (Error of the nonlinear term as a multiple of the run-time-plan kernels', with 9 and
  // without: 576 modes 1.12 and 1.06, 864 1.09 and 1.04, 288 1.06 and 1.01; a step took 3, 2 and 7 % longer, and
  // up to 5 % at lengths below, where both errors are alike: those keep it.)
  auto noise = [&](const std::vector<int>& r) { return fx || N < 512 ? 0 : (int)std::count(r.begin(), r.end(), 9); };
  auto padding = [&](const std::vector<int>& r) {
    if (fx) return 0;
    for (int v : r)
      if (v % 2) return 0;
    return 48 / r[0];
  };
  auto go = [&](auto&& self, int rest, int from) -> void {
    if (rest == 1) {
      int sum = 0;
      for (int r : cur) sum += r;
      const int a = 100 * noise(cur) + padding(cur), b = best.empty() ? 0 : 100 * noise(best) + padding(best);
      if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && (a < b || (a == b && sum < best_sum)))) {
        best = cur;
        best_sum = sum;
      }
      return;
    }
    if (!best.empty() && cur.size() + 1 > best.size()) return;
    for (int k = from; k < 8; ++k)
      if (rest % all[k] == 0) {
        cur.push_back(all[k]);
        self(self, rest / all[k], k);
        cur.pop_back();
      }
  };
  go(go, N, fx ? 2 : 0);
  if (fx) return best;
  // last: an odd radix, which needs no padding (mwf_zwarp.cuh), else the largest
  size_t last = 0;
  for (size_t k = 0; k < best.size(); ++k)
    if (best[k] % 2) { last = k; break; }
  std::swap(best[last], best.back());
  return best;
}
int inplace_line(int N) {                    // padded line length
  const int last = inplace_radices(N, false).back();
  return last % 2 ? N : N + N / last;
}

// Plan of the in-place transforms of length N, its stage twiddles (from w, the table of
// e^{-2 pi i t/(3N)}) and the element that each position of a digit-reversed line holds.
template <typename W>
bool make_fx_plan(int N, const std::vector<W>& w, bool fx, FxPlan& pl, std::vector<W>& tw, std::vector<unsigned short>& rev) {
  if (!is_23_smooth(N) || N < 2) return false;
  const std::vector<int> rad = inplace_radices(N, fx);
  if ((int)rad.size() > MWF_MAX_STAGES) return false;
  memset(&pl, 0, sizeof pl);
  pl.N = N;
  pl.nst = (int)rad.size();
  tw.clear();
  int span = N;
  for (int s = 0; s < pl.nst; ++s) {
    const int st = span / rad[s];
    pl.radix[s] = rad[s];
    pl.stride[s] = st;
    pl.tw_off[s] = (int)tw.size();
    pl.fnb[s] = make_fastdiv(N / rad[s]);
    pl.fst[s] = make_fastdiv(st);
    if (st > 1)
      for (int r = 1; r < rad[s]; ++r)
        for (int j = 0; j < st; ++j) tw.push_back(w[(size_t)3 * (j * r * (N / span) % N)]);
    span = st;
  }
  const int pad = rad.back() % 2 ? 0 : rad.back();
  pl.fpad = pad ? make_fastdiv(pad) : FastDiv{0, 2};      // without padding: quotient 0
  auto place = [&](int i) { return pad ? i + i / pad : i; };
  pl.LS = place(N);
  for (int s = 0; s < pl.nst; ++s) {
    pl.step[s] = pl.stride[s] == 1 ? 1 : place(pl.stride[s]);
    pl.bstep[s] = place(pl.stride[s] * rad[s]);
  }
  rev.assign(N, 0);
  for (int p = 0; p < N; ++p) {
    int q = 0, span_q = 1;
    for (int s = 0; s < pl.nst; ++s) {
      q += (p / pl.stride[s]) % pl.radix[s] * span_q;
      span_q *= pl.radix[s];
    }
    rev[p] = (unsigned short)q;
  }
  return span == 1;
}

// Tables of the fixed-point transforms of a run: e^{-2 pi i t/3N} and the plan of both lengths.
struct FxTables {
  std::vector<int4> wX, wZ, tM, tQ;
  std::vector<unsigned short> rev, revQ;
};
bool make_fx_tables(int MM, int NN, const std::vector<long double>& vX, const std::vector<long double>& vZ, RunDesc& D, FxTables& t) {
  auto table = [](const std::vector<long double>& v, std::vector<int4>& w) {
    w.resize(v.size() / 2);
    for (size_t j = 0; j < w.size(); ++j) w[j] = fx_twiddle(&v[2 * j]);
  };
  table(vX, t.wX);
  table(vZ, t.wZ);
  return make_fx_plan(MM, t.wX, true, D.fx_planM, t.tM, t.rev) && make_fx_plan(NN, t.wZ, true, D.fx_planQ, t.tQ, t.revQ) &&
         t.tM.size() <= (size_t)MM && t.tQ.size() <= (size_t)NN;
}

// var_precompute tables (variables.f90:516-531) and var_LHSRHS (variables.f90:565-597) in
// the reference's loop order, stored in the device layout [n][k][m].
void lhsrhs(const mwf_run_desc& d, std::vector<double>& inv_lhs, std::vector<double>& rhs) {
  const int MM = d.MM, NN = d.NN, K0 = d.K0, M = 2 * (MM - 1) + 1, K = 2 * K0 - 1;
  const double beta = 3.1415926535897931 / 2.0;
  std::vector<double> m2(M), n2(NN), k2(K0);
  for (int m = 0; m < MM; ++m) {
    if (m > 0) m2[M - m] = -d.alpha * m * d.alpha * m;
    m2[m] = -d.alpha * m * d.alpha * m;
  }
  for (int n = 0; n < NN; ++n) n2[n] = -d.gamma * n * d.gamma * n;
  for (int k = 0; k < K0; ++k) k2[k] = -k * k * beta * beta;
  std::vector<double> L((size_t)NN * K * M), R((size_t)NN * K * M);
  auto at = [&](std::vector<double>& a, int k, int m, int n) -> double& { return a[((size_t)n * K + k) * M + m]; };
  for (int n = 0; n < NN; ++n)
    for (int m = 0; m < M; ++m)
      for (int k = 0; k < K0; ++k) {
        const int a = k, b = k + K0 - 1;
        const double lap = m2[m] + k2[k] + n2[n];
        const double hlap = m2[m] + n2[n];
        const double ilap16 = d.hypo / (m2[m] + k2[k] + n2[n]);
        double tvl;
        if (d.dragall || k == 0) tvl = 1.0 - d.dt * (lap / d.Re + ilap16 - d.drag);
        else tvl = 1.0 - d.dt * (lap / d.Re + ilap16);
        if (m == 0 && n == 0) {
          at(L, a, m, n) = tvl;
          at(L, b, m, n) = tvl;
          at(R, a, m, n) = 1.0;
          at(R, b, m, n) = 1.0;
          at(L, 0, m, n) = 1.0;
          at(R, 0, m, n) = 0.0;
        } else {
          at(L, a, m, n) = tvl * hlap;
          if (d.dragall) at(L, b, m, n) = tvl * hlap * lap + d.dt * (d.vdrag - d.drag) * hlap * hlap;
          else at(L, b, m, n) = tvl * hlap * lap;
          at(R, a, m, n) = hlap;
          at(R, b, m, n) = hlap * lap;
        }
      }
  inv_lhs.resize(L.size());
  for (size_t i = 0; i < L.size(); ++i) inv_lhs[i] = 1.0 / L[i];
  rhs.swap(R);
}

struct RunHost {
  mwf_run_desc d;
  int K, KK, M, X, Z;
  size_t csz;        // complex elements of c
  size_t off_c, off_onl, off_ilhs, off_rhs, off_T, off_NLT, off_twX, off_twQ, off_twZ, off_nst;
  int n_diag_xf, n_diag_z;   // work items of the physical-space diagnostic
  int xf_nb, xi_nb, z_lx;
  int z_ppt, z_nt;
  int x_nt;          // block size of the x passes
  int x_radix, z_radix;
  int zb_lx = 0;     // x lines per item of the batched FP32 z pass (0: z_nonlinear_kernel)
  int xbf_nb = 0, xbi_nb = 0;   // columns per item of the subset-split FP32 x passes (0: not used)
  bool persist = false;         // all three passes batched: the run steps in the persistent kernel
  int active = 1;    // host copy of RunDesc::active
  // FP32 z pass with a warp per line (mwf_zwarp.cuh): lines per item (0: not used), subsets at once,
  // block size
  int zw_lines = 0, zw_ns = 0, zw_nt = 0;
  size_t off_zw = 0;
  // FP32 x passes with a warp per line (mwf_xwarp.cuh): columns per item (0: not used), field and
  // derivative at once or in turn, block sizes
  int xw_fnb = 0, xw_inb = 0, xw_nd = 0, xw_fnt = 0, xw_int = 0;
  size_t off_xw = 0;
  // FP64 in fixed point (mwf_fxpass.cuh): columns and block sizes of the x passes, lines and block
  // size of the z pass
  bool fx = false;
  int fx_nb = 0, fx_xi_nb = 0, fx_lines = 0, fx_nblk = 0, fx_tab = 0, fx_group = 0;
  int fx_z_nt = 0, fx_xi_nt = 0;      // the x forward always fits half an SM: 256
  size_t off_fx = 0;
  struct FxOff { size_t twX, twZ, twM, twQ, gn, mp, ms, rev, revQ, colE, blkE, rowE, minE, rowP, end; };
  FxOff fx_off() const {
    FxOff o;
    size_t a = off_fx;
    auto put = [&](size_t bytes) { const size_t at = a; a = (a + bytes + 255) / 256 * 256; return at; };
    o.twX = put(16 * (size_t)X);
    o.twZ = put(16 * (size_t)Z);
    o.twM = put(16 * (size_t)d.MM);           // a length N has fewer than N stage twiddles
    o.twQ = put(16 * (size_t)d.NN);
    o.gn = put(16 * (size_t)d.NN);
    o.mp = put(16 * (size_t)4 * d.MM);
    o.ms = put(16 * (size_t)d.MM);
    o.rev = put(2 * (size_t)d.MM);
    o.revQ = put(2 * (size_t)d.NN);
    o.colE = put(4 * (size_t)2 * KK * d.NN);
    o.blkE = put(4 * (size_t)2 * KK * fx_nblk);
    o.rowE = put(4 * (size_t)3 * KK * X);
    o.minE = put(4 * (size_t)KK);
    o.rowP = put(4 * (size_t)2 * KK * X * fx_nblk);
    o.end = a;
    return o;
  }
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Items of one launch: each takes up to *width of a run's `lines`, `per` times.
struct ItemWidth {
  int* width;
  int lines, per;
  bool fixed;        // by a tuning knob
};
// plan_run takes the widest items that fit, which read and set up the least per line.  A launch whose runs
// together give fewer than `slots` of them leaves SMs without one while each item takes its lines
// in turn, so there the narrowest width that still makes one round is taken.
void spread_items(std::vector<ItemWidth>& v, int slots, bool pow2) {
  int widest = 1;
  for (const ItemWidth& x : v) widest = std::max(widest, *x.width);
  int w = 1;
  for (; w < widest; w = pow2 ? 2 * w : w + 1) {
    long items = 0;
    for (const ItemWidth& x : v) {
      const int own = x.fixed ? *x.width : std::min(w, *x.width);
      items += (long)((x.lines + own - 1) / own) * x.per;
    }
    if (items <= slots) break;
  }
  for (const ItemWidth& x : v)
    if (!x.fixed) *x.width = std::min(w, *x.width);
}

// Tiling of one run; returns false if the run does not fit the kernels' shapes.
bool plan_run(RunHost& r, const char*& why) {
  const mwf_run_desc& d = r.d;
  if (d.K0 != 4 && d.K0 != 6) { why = "K0 must be 4 (M4) or 6 (M6)"; return false; }
  if (d.MM < 2 || d.NN < 2) { why = "MM and NN must be >= 2"; return false; }
  if (!is_23_smooth(d.MM) || !is_23_smooth(d.NN)) { why = "MM and NN must be of the form 2^a 3^b"; return false; }
  r.K = 2 * d.K0 - 1;
  r.KK = 3 * d.K0 - 1;
  r.M = 2 * (d.MM - 1) + 1;
  r.X = 3 * d.MM;
  r.Z = 3 * d.NN;
  if (r.X > kMaxLen) { why = "3*MM exceeds the longest supported x line (4096)"; return false; }
  if (d.NN > kMaxNN) { why = "NN exceeds the longest supported z half-line (1024)"; return false; }
  if (d.precision != MWF_FP64 && d.precision != MWF_FP32) { why = "precision must be MWF_FP64 or MWF_FP32"; return false; }
  const size_t cb = d.precision == MWF_FP64 ? 16 : 8;
  // x forward: nb*X <= VPT*threads, smem <= limit; equal tiles
  r.x_nt = xpass_threads(d.precision, r.X);
  const int xfv = xf_vpt(d.precision);
  // the FP64 x forward also holds its wavenumber tables in static shared memory
  const size_t xf_smem = kSmemLimit - (d.precision == MWF_FP64 ? kXTabBytes : 0);
  int nbmax = std::min(xfv * r.x_nt / r.X, (int)(xf_smem / (r.X * cb * 9 / 8 + cb)));
  nbmax = std::max(1, std::min(nbmax, d.NN));
  if (nbmax * r.X > xfv * r.x_nt) { why = "x line too long for the x-forward pass"; return false; }
  r.xf_nb = d.NN / ((d.NN + nbmax - 1) / nbmax);
  while (r.xf_nb > 1 && d.NN % r.xf_nb) --r.xf_nb;
  // FP32 runs whose MM has a compile-time plan use the subset-split x passes unless an x radix
  // cap is given (which selects x_forward_kernel / x_inverse_kernel and their run-time plans);
  // the column knobs then apply to them
  const bool xb = d.precision == MWF_FP32 && d.x_radix == 0 && xb_supported(d.MM);
  r.xbf_nb = r.xbi_nb = 0;
  if (xb) {
    auto widest = [&](size_t (*smem)(int, int), size_t budget) {
      int nb = 1;
      while (nb < 8 && nb < d.NN && smem(d.MM, nb + 1) <= budget) ++nb;
      return nb;
    };
    const size_t fbudget = zb_smem_budget(kXfBlocks), ibudget = zb_smem_budget(kXiBlocks);
    const int fmax = widest(xbf_smem, fbudget), imax = widest(xbi_smem, ibudget);
    if (xbf_smem(d.MM, 1) > fbudget || xbi_smem(d.MM, 1) > ibudget) { why = "x line too long for the x passes"; return false; }
    r.xbf_nb = fmax;
    r.xbi_nb = imax;
    if (d.xf_cols) {
      if (d.xf_cols < 1 || d.xf_cols > std::min(fmax, d.NN)) { why = "xf_cols out of range for this run"; return false; }
      r.xbf_nb = d.xf_cols;
    }
    if (d.xi_cols) {
      if (d.xi_cols < 1 || d.xi_cols > std::min(imax, d.NN)) { why = "xi_cols out of range for this run"; return false; }
      r.xbi_nb = d.xi_cols;
    }
  }
  if (d.xf_cols && !xb) {
    if (d.xf_cols < 1 || d.xf_cols > nbmax) { why = "xf_cols out of range for this run"; return false; }
    r.xf_nb = d.xf_cols;
  }
  // x inverse: nb*X <= VPT*threads per field, three fields resident
  nbmax = std::min(kXiVpt * r.x_nt / r.X, (int)(kSmemLimit / (3 * r.X * cb * 9 / 8 + cb)));
  nbmax = std::max(1, std::min(nbmax, d.NN));
  if (nbmax * r.X > kXiVpt * r.x_nt) { why = "x line too long for the x-inverse pass"; return false; }
  r.xi_nb = d.NN / ((d.NN + nbmax - 1) / nbmax);
  while (r.xi_nb > 1 && d.NN % r.xi_nb) --r.xi_nb;
  if (d.xi_cols && !xb) {
    if (d.xi_cols < 1 || d.xi_cols > nbmax) { why = "xi_cols out of range for this run"; return false; }
    r.xi_nb = d.xi_cols;
  }
  // z pass: points per CTA = threads * points-per-thread >= NN
  r.z_ppt = d.NN <= kZThreads ? 1 : 2;
  r.z_nt = (d.precision == MWF_FP32 && d.NN <= kZThreadsSmall) ? kZThreadsSmall : kZThreads;
  if (d.K0 == 6 && d.precision == MWF_FP64 && r.z_ppt == 2) {
    why = "M6 in FP64 supports NN <= 512";
    return false;
  }
  r.z_lx = std::max(1, r.z_nt * r.z_ppt / d.NN);
  r.z_lx = std::min(r.z_lx, r.X);
  // FP32 runs whose z line length has a compile-time plan use the batched z pass unless a z
  // radix cap is given (which selects z_nonlinear_kernel and its run-time plans)
  r.zb_lx = 0;
  if (d.precision == MWF_FP32 && d.z_radix == 0 && zb_supported(d.K0, d.NN)) {
    const size_t budget = zb_smem_budget(zb_blocks_per_sm(d.K0, d.NN));
    int L = 1;
    while (L < r.X && zb_smem(d.K0, d.NN, L + 1) <= budget) ++L;
    if (d.z_lines) {
      if (d.z_lines < 1 || d.z_lines > L) { why = "z_lines out of range for this run"; return false; }
      L = d.z_lines;
    }
    r.zb_lx = L;
  } else if (d.z_lines) {
    if (d.z_lines < 1 || d.z_lines > r.z_lx) { why = "z_lines out of range for this run"; return false; }
    r.z_lx = d.z_lines;
  }
  // largest radix: the kernels' compile-time caps (x: 12 FP64 / 16 FP32; z: 8 / 12)
  const int xcap = d.precision == MWF_FP64 ? 12 : 16, zcap = d.precision == MWF_FP64 ? 8 : 12;
  auto radix_ok = [](int v, int cap) { return v == 0 || ((v == 8 || v == 12 || v == 16) && v <= cap); };
  if (!radix_ok(d.x_radix, xcap) || !radix_ok(d.z_radix, zcap)) { why = "x_radix/z_radix must be 8, 12 or 16 within the pass caps"; return false; }
  r.x_radix = d.x_radix ? d.x_radix : xcap;
  r.z_radix = d.z_radix ? d.z_radix : zcap;
  // FP32 runs that neither the batched z pass takes nor a knob directs to z_nonlinear_kernel: a warp
  // per line
  r.zw_lines = 0;
  if (d.precision == MWF_FP32 && !r.zb_lx && !d.z_radix && !d.z_lines) {
    const int LS = inplace_line(d.NN);
    auto need = [&](int L) { return zw_smem(d.K0, d.NN, LS, r.zw_ns, L); };
    r.zw_ns = 3;
    if (need(1) > zb_smem_budget(1)) r.zw_ns = 1;
    if (need(1) <= zb_smem_budget(1)) {
      r.zw_nt = need(1) <= zb_smem_budget(2) ? 256 : (d.K0 == 6 && r.zw_ns == 3 ? 512 : 576);
      const size_t zbud = zb_smem_budget(r.zw_nt == 256 ? 2 : 1);
      const int g = std::max(1, 128 / d.NN);    // lines of a warp's task
      int L = 1;
      while (L < r.X && L * d.NN < 512 && need(L + 1) <= zbud) ++L;
      r.zw_lines = L > g ? L / g * g : L;
    }
  }
  r.xw_fnb = r.xw_inb = 0;
  if (d.precision == MWF_FP32 && !xb && !d.x_radix && !d.xf_cols && !d.xi_cols) {
    const int LS = inplace_line(d.MM);
    const size_t half = zb_smem_budget(2), whole = zb_smem_budget(1);
    // eight columns at most; narrower where field and derivative do not fit half an SM together,
    // and then, from four columns (a sector of T) down, one after the other
    r.xw_nd = 2;
    r.xw_fnb = 8;
    while (r.xw_fnb > 4 && (xw_fsmem(d.MM, LS, 2, r.xw_fnb) > half || r.xw_fnb / 2 >= d.NN)) r.xw_fnb /= 2;
    if (xw_fsmem(d.MM, LS, 2, r.xw_fnb) > half) r.xw_nd = 1;
    while (r.xw_fnb > 1 && xw_fsmem(d.MM, LS, r.xw_nd, r.xw_fnb) > half) r.xw_fnb /= 2;
    r.xw_fnt = xw_fsmem(d.MM, LS, r.xw_nd, r.xw_fnb) <= half ? 256 : 512;
    r.xw_inb = 8;
    while (r.xw_inb > 1 && (xw_ismem(d.MM, LS, r.xw_inb) > (r.xw_inb <= 4 ? whole : half) || r.xw_inb / 2 >= d.NN)) r.xw_inb /= 2;
    r.xw_int = xw_ismem(d.MM, LS, r.xw_inb) <= half ? 256 : 512;
  }
  // FP64 runs without tuning knobs step in 64-bit fixed point (mwf_fxpass.cuh) where one line of
  // the z pass, all transforms of a z-subset, fits a CTA; the knobs belong to the FP64-arithmetic
  // kernels, which the longest z lines (M4 beyond NN = 768) keep
  r.fx = d.precision == MWF_FP64 && !d.xf_cols && !d.xi_cols && !d.z_lines && !d.x_radix && !d.z_radix &&
         fx_z_smem(d.K0, d.NN, 1) <= zb_smem_budget(1);
  if (r.fx) {
    const size_t half = zb_smem_budget(2) - 1408, whole = zb_smem_budget(1) - 1408;   // the x passes' static arrays
    const int slots = 2 * 152;                // CTAs of 256 threads that the chip holds
    auto items = [&](int nb, int per) { return (d.NN + nb - 1) / nb * per; };
    // widest column blocks (whole sectors of T) that still give every slot an item
    r.fx_nb = kFxMaxCols;
    while (r.fx_nb > 1 && (fx_xf_smem(d.MM, r.fx_nb) > half || (r.fx_nb > 2 && items(r.fx_nb, 2 * r.KK) < slots))) r.fx_nb /= 2;
    r.fx_nblk = (d.NN + r.fx_nb - 1) / r.fx_nb + 1;    // and column n = 0 by itself
    r.fx_xi_nb = kFxMaxCols;
    while (r.fx_xi_nb > 1 && (fx_xi_smem(d.MM, r.fx_xi_nb) > (r.fx_xi_nb == 2 ? whole : half) ||
                              (r.fx_xi_nb > 2 && items(r.fx_xi_nb, d.K0) < slots))) r.fx_xi_nb /= 2;
    r.fx_xi_nt = fx_xi_smem(d.MM, r.fx_xi_nb) <= half ? 256 : 512;
    // z pass: block size (256 threads, two CTAs per SM; 512; for M4 also 544, a warp for each of its 17
    // lines), lines per item and lines of a warp's task, by an estimate of a CTA's time -- the rounds
    // that its warps make over fill, transforms and points, in thousands of cycles as measured on
    // NN = 48 and 512 -- times the waves of CTAs
    const int ntr = (3 * r.KK + 1) / 2, npair = (r.KK + 1) / 2, zslots = (d.NN + 1) / 2;
    const std::vector<int> rad = inplace_radices(d.NN, true);
    const int g0 = std::max(1, 256 / d.NN);
    auto up = [](long a, long b) { return (a + b - 1) / b; };
    double best = -1.0;
    for (int nt : {256, 512, 544}) {
      if (nt == 544 && d.K0 != 4) continue;
      const long warps = nt / 32, per_sm = nt == 256 ? 2 : 1;
      for (int L = 1; L <= 2 * g0 + 1 && L <= r.X; ++L) {
        if (fx_z_smem(d.K0, d.NN, L) > zb_smem_budget((int)per_sm)) continue;
        for (int G = 1; G <= std::min(L, g0 + 1); ++G) {
          const long groups = up(L, G), fill = up((long)G * zslots, 32);
          double fft = 0.0;                     // a butterfly of radix 8 as the unit
          for (int q : rad) fft += up((long)G * d.NN / q, 32) * (q / 8.0 + 0.2);
          const double cta = up(ntr * groups, warps) * (2.0 * fill + 2.2 * fft) +
                             up(npair * groups, warps) * (1.0 * fill + 2.0 * fft + 2.0) +
                             up((long)L * d.NN, nt) * (d.K0 == 4 ? 10.0 : 30.0) + 8.0;
          const double cost = cta * up(up(r.X, L) * 3, 152 * per_sm);
          if (best < 0.0 || cost < best) {
            best = cost;
            r.fx_z_nt = nt;
            r.fx_lines = L;
            r.fx_group = G;
          }
        }
      }
    }
    r.fx_tab = 2;
    while (r.fx_tab > 0 && fx_z_smem(d.K0, d.NN, r.fx_lines, r.fx_tab) > zb_smem_budget(r.fx_z_nt == 256 ? 2 : 1)) --r.fx_tab;
  }
  r.n_diag_xf = ((d.NN + r.xf_nb - 1) / r.xf_nb) * r.KK;
  r.n_diag_z = ((r.X + r.z_lx - 1) / r.z_lx) * 3;
  return true;
}

size_t run_bytes(RunHost& r, size_t base) {
  const size_t cb = r.d.precision == MWF_FP64 ? 16 : 8;
  size_t o = base;
  r.csz = (size_t)r.K * r.M * r.d.NN;
  r.off_c = o; o = align_up(o + r.csz * cb, 256);
  r.off_onl = o; o = align_up(o + r.csz * cb, 256);
  r.off_ilhs = o; o = align_up(o + r.csz * 8, 256);
  r.off_rhs = o; o = align_up(o + r.csz * 8, 256);
  r.off_T = o; o = align_up(o + (size_t)2 * r.KK * r.X * r.d.NN * cb, 256);
  r.off_NLT = o; o = align_up(o + (size_t)3 * r.KK * r.X * r.d.NN * cb, 256);   // one partial per z-subset
  r.off_twX = o; o = align_up(o + (size_t)r.X * cb, 256);
  r.off_twQ = o; o = align_up(o + (size_t)r.d.NN * cb, 256);
  r.off_twZ = o; o = align_up(o + (size_t)r.Z * cb, 256);
  r.off_nst = o; o = align_up(o + sizeof(int), 256);
  if (r.zw_lines) {
    r.off_zw = o;
    o = align_up(o + sizeof(float2) * (size_t)r.d.NN, 256);
  }
  if (r.xw_fnb) {
    r.off_xw = o;
    o = align_up(o + sizeof(float2) * (size_t)r.d.MM, 256);
    o = align_up(o + sizeof(unsigned short) * (size_t)r.d.MM, 256);
  }
  if (r.fx) {
    r.off_fx = o;
    o = r.fx_off().end;
  }
  return o;
}

struct Launch {
  int kind;       // 0 x-forward, 1 z pass, 2 x-inverse
  int prec, K0, ppt, nt;
  size_t smem;
  size_t item_off; // offset into the device item array
  int nitems;
  int zbQ = 0;     // z pass: 0 = z_nonlinear_kernel, else the batched FP32 z pass for NN = zbQ
  int xbMM = 0;    // x passes: 0 = x_forward_kernel / x_inverse_kernel, else the subset-split
                   // FP32 kernels for MM = xbMM
  bool fx = false;              // FP64 passes in fixed point
  int zw_ns = 0;                // FP32 z pass with a warp per line: subsets at once
  bool xw = false;              // FP32 x passes with a warp per line
  bool persist_group = false;   // its runs can step in the persistent kernel instead (step mode)
};

cudaError_t launch_pass(const Launch& L, const RunDesc* runs, const WorkItem* items, int* err, cudaStream_t st) {
  if (L.fx) {
    if (L.kind == 0) return launch_x_forward_fx(runs, items, L.nitems, L.smem, st);
    if (L.kind == 1) return launch_z_fx(L.K0, L.nt, runs, items, L.nitems, L.smem, st);
    return launch_x_inverse_fx(L.nt, runs, items, L.nitems, L.smem, st);
  }
  if (L.xw)
    return L.kind == 0 ? launch_x_forward_warp(L.nt, runs, items, L.nitems, L.smem, st)
                       : launch_x_inverse_warp(L.nt, runs, items, L.nitems, L.smem, st);
  if (L.zw_ns) return launch_z_warp(L.K0, L.zw_ns, L.nt, runs, items, L.nitems, L.smem, st);
  if (L.kind == 0 && L.xbMM) return launch_x_forward_batched(L.xbMM, runs, items, L.nitems, L.smem, err, st);
  if (L.kind == 2 && L.xbMM) return launch_x_inverse_batched(L.xbMM, runs, items, L.nitems, L.smem, err, st);
  if (L.kind == 0)
    return L.prec == 0 ? launch_x_forward_f64(L.nt, runs, items, L.nitems, L.smem, err, st)
                       : launch_x_forward_f32(L.nt, runs, items, L.nitems, L.smem, err, st);
  if (L.kind == 1) {
    if (L.zbQ) return launch_z_batched(L.K0, L.zbQ, runs, items, L.nitems, L.smem, err, st);
    return L.prec == 0 ? launch_z_nonlinear_f64(L.K0, L.ppt, L.nt, runs, items, L.nitems, L.smem, err, st)
                       : launch_z_nonlinear_f32(L.K0, L.ppt, L.nt, runs, items, L.nitems, L.smem, err, st);
  }
  return L.prec == 0 ? launch_x_inverse_f64(L.nt, runs, items, L.nitems, L.smem, err, st)
                     : launch_x_inverse_f32(L.nt, runs, items, L.nitems, L.smem, err, st);
}

}  // namespace

struct mwf_handle {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::vector<RunHost> runs;
  unsigned char* arena = nullptr;
  size_t arena_bytes = 0;
  RunDesc* d_runs = nullptr;
  WorkItem* d_items = nullptr;
  WorkItem* d_diag_items = nullptr;  // scratch for one run's diagnostic work items
  int* d_err = nullptr;
  int* d_flag = nullptr;
  unsigned* d_ticket = nullptr;  // blocks of the energy kernel that have finished
  double* d_partial = nullptr;
  HostOut* h_out = nullptr;      // pinned host memory that kernels write a call's outcome to
  double* d_stage = nullptr;     // 2 * max(csz) doubles for state copies
  size_t stage_elems = 0;
  std::vector<Launch> launches;
  size_t off_nst_all = 0;            // arena offset of the runs' Euler-start flags (one int each)
  // persistent FP32 step: its items, counters (cleared before every launch), shared memory, grid
  void* d_pitems = nullptr;
  int n_pitems = 0;
  int* d_counters = nullptr;
  size_t counters_bytes = 0;
  size_t persist_smem = 0;
  int persist_grid = 0;
  bool persist_mode = false;         // step with the persistent kernel (mwf_set_persistent)
  bool any_sym = false;
  bool euler_pending = true;          // a run's Euler-start flag may be set: the next step clears it
  cudaGraphExec_t graph1 = nullptr;   // one step
  cudaGraphExec_t graphG = nullptr;   // kGraphSteps steps
  static constexpr int kGraphSteps = 16;
  static constexpr int kEnergyParts = 2432;  // blocks of the energy kernel: sixteen per SM
};

namespace {

// One step on the handle's stream; clear_euler: with the reset of the runs' Euler-start flags, which
// only the first step after a flag was set needs (the graphs leave it out: a memset node cost a
// small run's step about 2 us).
int enqueue_step(mwf_handle* h, bool clear_euler) {
  cudaStream_t st = h->stream;
  if (h->any_sym) {
    for (size_t i = 0; i < h->runs.size(); ++i) {
      const RunHost& r = h->runs[i];
      const int modes[3] = {r.d.reflect, r.d.uvreflect, r.d.wreflect};
      for (int mode = 0; mode < 3; ++mode) {
        if (!modes[mode]) continue;
        cudaError_t e = r.d.precision == MWF_FP64
                            ? launch_imposesym_f64(h->d_runs, (int)i, mode, r.M, r.d.NN, st)
                            : launch_imposesym_f32(h->d_runs, (int)i, mode, r.M, r.d.NN, st);
        if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "imposesym launch: %s", cudaGetErrorString(e));
      }
    }
  }
  const bool persist = h->persist_mode && h->n_pitems;
  if (persist) {
    cudaError_t e = cudaMemsetAsync(h->d_counters, 0, h->counters_bytes, st);
    if (e == cudaSuccess)
      e = launch_persistent_step(h->d_runs, h->d_pitems, h->n_pitems, h->d_counters, h->persist_smem,
                                 h->persist_grid, h->d_err, st);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "persistent step launch: %s", cudaGetErrorString(e));
  }
  for (const Launch& L : h->launches) {
    if (persist && L.persist_group) continue;
    cudaError_t e = launch_pass(L, h->d_runs, h->d_items + L.item_off, h->d_err, st);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "pass %d launch: %s", L.kind, cudaGetErrorString(e));
  }
  // the Euler start applies to one step only (velocity.f90:24-27)
  if (clear_euler) {
    const cudaError_t e = cudaMemsetAsync(h->arena + h->off_nst_all, 0, sizeof(int) * h->runs.size(), st);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "nst reset: %s", cudaGetErrorString(e));
  }
  return MWF_OK;
}

int build_graph(mwf_handle* h, int steps, cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
  int rc = MWF_OK;
  for (int s = 0; s < steps && rc == MWF_OK; ++s) rc = enqueue_step(h, false);
  cudaError_t e = cudaStreamEndCapture(h->stream, &g);
  if (rc != MWF_OK) { if (g) cudaGraphDestroy(g); return rc; }
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
  e = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
  return MWF_OK;
}

// x forward of the run's perturbation fields (without the base flow) by the kernels of the timestep;
// with_z: the items of the diagnostic z pass go up behind its own.
int diag_x_forward(mwf_handle* h, int run, bool with_z, cudaError_t& e) {
  const RunHost& r = h->runs[run];
  std::vector<WorkItem> items;
  items.reserve(r.n_diag_xf + r.n_diag_z);
  for (int n0 = 0; n0 < r.d.NN; n0 += r.xf_nb)
    for (int f = 0; f < r.KK; ++f) items.push_back(WorkItem{run, n0, f, 1});
  if (with_z)
    for (int x0 = 0; x0 < r.X; x0 += r.z_lx)
      for (int sub = 0; sub < 3; ++sub) items.push_back(WorkItem{run, x0, sub, 0});
  if ((int)items.size() != r.n_diag_xf + (with_z ? r.n_diag_z : 0)) return fail(MWF_ERR_DEVICE, "diagnostic item count mismatch");
  CK(cudaMemcpyAsync(h->d_diag_items, items.data(), sizeof(WorkItem) * items.size(), cudaMemcpyHostToDevice, h->stream));
  const size_t xfs = xpass_smem(r.d.precision, (size_t)r.xf_nb * r.X);
  e = r.d.precision == MWF_FP64 ? launch_x_forward_f64(r.x_nt, h->d_runs, h->d_diag_items, r.n_diag_xf, xfs, h->d_err, h->stream)
                                : launch_x_forward_f32(r.x_nt, h->d_runs, h->d_diag_items, r.n_diag_xf, xfs, h->d_err, h->stream);
  return MWF_OK;
}

// Wait for the stream; the error word is in h_out->err by then.
int finish_call(mwf_handle* h) {
  CK(cudaStreamSynchronize(h->stream));
  const int herr = h->h_out->err;
  if (herr) return fail(MWF_ERR_DEVICE, "kernel reported internal error flags 0x%x", herr);
  return MWF_OK;
}

int check_device_err(mwf_handle* h) {
  CK(cudaMemcpyAsync(&h->h_out->err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  return finish_call(h);
}

// Whether the device may access the n doubles at p in place: they lie within one pinned host
// allocation (or registration), at an address that the kernels' 8-byte accesses take (copies take any).
bool device_reads_host(const double* p, size_t n) {
  if (reinterpret_cast<uintptr_t>(p) % sizeof(double)) return false;
  static const auto attr = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<CUresult (*)(void*, CUpointer_attribute, CUdeviceptr)>(fn);
  }();
  if (!attr) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type != cudaMemoryTypeHost || a.devicePointer != (const void*)p) return false;
  CUdeviceptr start = 0;
  size_t size = 0;
  if (attr(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, (CUdeviceptr)p) != CUDA_SUCCESS ||
      attr(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, (CUdeviceptr)p) != CUDA_SUCCESS)
    return false;
  return (CUdeviceptr)p >= start && (CUdeviceptr)p + n * sizeof(double) <= start + size;
}

void free_handle(mwf_handle* h) {
  if (!h) return;
  if (h->graph1) cudaGraphExecDestroy(h->graph1);
  if (h->graphG) cudaGraphExecDestroy(h->graphG);
  if (h->arena) cudaFree(h->arena);
  if (h->h_out) cudaFreeHost(h->h_out);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

}  // namespace

extern "C" {

long long mwf_run_dof(const mwf_run_desc* d) {
  if (!d) return 0;
  return (long long)(2 * d->K0 - 1) * (2 * (d->MM - 1) + 1) * d->NN;
}

long long mwf_footprint_bytes(const mwf_run_desc* runs, int n_runs) {
  if (!runs || n_runs <= 0) return -1;
  size_t o = 0;
  size_t stage = 0;
  for (int i = 0; i < n_runs; ++i) {
    RunHost r;
    r.d = runs[i];
    const char* why = "";
    if (!plan_run(r, why)) return -1;
    o = run_bytes(r, o);
    stage = std::max(stage, r.csz);
  }
  return (long long)(o + 2 * stage * sizeof(double) + 4096 + (size_t)n_runs * sizeof(RunDesc));
}

int mwf_describe_run(const mwf_run_desc* d, mwf_run_plan* out) {
  if (!d || !out) return fail(MWF_ERR_ARG, "mwf_describe_run: null argument");
  RunHost r;
  r.d = *d;
  const char* why = "";
  if (!plan_run(r, why)) return fail(MWF_ERR_SIZE, "mwf_describe_run: %s", why);
  const int prec = d->precision == MWF_FP64 ? 0 : 1;
  mwf_run_plan p;
  memset(&p, 0, sizeof p);
  p.batched_x = r.xbf_nb ? 1 : 0;
  p.batched_z = r.zb_lx ? 1 : 0;
  if (p.batched_x) {
    p.xf_cols = r.xbf_nb;
    p.xi_cols = r.xbi_nb;
    p.xf_ctas_per_sm = kXfBlocks;
    p.xi_ctas_per_sm = kXiBlocks;
    p.xf_smem = (long long)xbf_smem(d->MM, r.xbf_nb);
    p.xi_smem = (long long)xbi_smem(d->MM, r.xbi_nb);
    p.xf_items = ((d->NN + r.xbf_nb - 1) / r.xbf_nb) * d->K0;
    p.xi_items = ((d->NN + r.xbi_nb - 1) / r.xbi_nb) * d->K0;
  } else if (r.xw_fnb) {
    const int LS = inplace_line(d->MM);
    p.xf_cols = r.xw_fnb;
    p.xi_cols = r.xw_inb;
    p.xf_smem = (long long)xw_fsmem(d->MM, LS, r.xw_nd, r.xw_fnb);
    p.xi_smem = (long long)xw_ismem(d->MM, LS, r.xw_inb);
    p.xf_items = ((d->NN + r.xw_fnb - 1) / r.xw_fnb) * d->K0;
    p.xi_items = ((d->NN + r.xw_inb - 1) / r.xw_inb) * d->K0;
  } else if (r.fx) {
    p.xf_cols = r.fx_nb;
    p.xi_cols = r.fx_xi_nb;
    p.xf_smem = (long long)fx_xf_smem(d->MM, r.fx_nb);
    p.xi_smem = (long long)fx_xi_smem(d->MM, r.fx_xi_nb);
    p.xf_items = (r.fx_nblk - 1) * 2 * r.KK;
    p.xi_items = ((d->NN + r.fx_xi_nb - 1) / r.fx_xi_nb) * d->K0;
  } else {
    p.xf_cols = r.xf_nb;
    p.xi_cols = r.xi_nb;
    p.xf_smem = (long long)xpass_smem(prec, (size_t)r.xf_nb * r.X);
    p.xi_smem = (long long)xpass_smem(prec, (size_t)3 * r.xi_nb * r.X);
    p.xf_items = ((d->NN + r.xf_nb - 1) / r.xf_nb) * 2 * r.KK;
    p.xi_items = ((d->NN + r.xi_nb - 1) / r.xi_nb) * d->K0;
  }
  if (p.batched_z) {
    p.z_lines = r.zb_lx;
    p.z_ctas_per_sm = zb_blocks_per_sm(d->K0, d->NN);
    p.z_smem = (long long)zb_smem(d->K0, d->NN, r.zb_lx);
    p.z_items = (r.X + r.zb_lx - 1) / r.zb_lx;
  } else if (r.zw_lines) {
    p.z_lines = r.zw_lines;
    p.z_smem = (long long)zw_smem(d->K0, d->NN, inplace_line(d->NN), r.zw_ns, r.zw_lines);
    p.z_items = (r.X + r.zw_lines - 1) / r.zw_lines;
  } else if (r.fx) {
    p.z_lines = r.fx_lines;
    p.z_smem = (long long)fx_z_smem(d->K0, d->NN, r.fx_lines, r.fx_tab);
    p.z_items = ((r.X + r.fx_lines - 1) / r.fx_lines) * 3;
  } else {
    p.z_lines = r.z_lx;
    p.z_smem = (long long)zpass_smem(prec, d->K0, r.z_ppt, r.z_nt);
    p.z_items = ((r.X + r.z_lx - 1) / r.z_lx) * (zpass_summed(prec) ? 1 : 3);
  }
  *out = p;
  return MWF_OK;
}

int mwf_create(const mwf_run_desc* runs, int n_runs, int device, mwf_handle** out) {
  if (!runs || n_runs <= 0 || !out) return fail(MWF_ERR_ARG, "mwf_create: null argument or n_runs <= 0");
  *out = nullptr;
  mwf_handle* h = new mwf_handle();
  h->device = device;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    free_handle(h);
    return fail(MWF_ERR_CUDA, "mwf_create: no CUDA device");
  }
  if (device < 0 || device >= ndev) { free_handle(h); return fail(MWF_ERR_ARG, "mwf_create: bad device %d", device); }
  if (cudaSetDevice(device) != cudaSuccess) { free_handle(h); return fail(MWF_ERR_CUDA, "cudaSetDevice failed"); }
  h->runs.resize(n_runs);
  size_t o = 0;
  for (int i = 0; i < n_runs; ++i) {
    RunHost& r = h->runs[i];
    r.d = runs[i];
    const char* why = "";
    if (!plan_run(r, why)) { free_handle(h); return fail(MWF_ERR_SIZE, "run %d: %s", i, why); }
    if ((r.d.reflect || r.d.uvreflect || r.d.wreflect) && r.d.K0 != 4) {
      free_handle(h);
      return fail(MWF_ERR_ARG, "run %d: the reference defines the symmetry masks for K0 = 4 only", i);
    }
    if (r.d.reflect || r.d.uvreflect || r.d.wreflect) h->any_sym = true;
    if (!(r.d.dt > 0) || !(r.d.Re > 0)) { free_handle(h); return fail(MWF_ERR_ARG, "run %d: dt and Re must be > 0", i); }
    o = run_bytes(r, o);
    h->stage_elems = std::max(h->stage_elems, r.csz);
  }
  // the Euler-start flags of all runs side by side, so one memset clears them (enqueue_step)
  const size_t off_nst_all = o; o = align_up(o + sizeof(int) * n_runs, 256);
  for (int i = 0; i < n_runs; ++i) h->runs[i].off_nst = off_nst_all + sizeof(int) * i;
  h->off_nst_all = off_nst_all;
  const size_t off_runs = o; o = align_up(o + sizeof(RunDesc) * n_runs, 256);
  // work items
  std::vector<WorkItem> items;
  // group launches: x-forward per precision, z pass per (precision, K0, threads), x-inverse per precision
  static const int kXbSizes[] = {32, 48, 64, 96, 128, 192, 256};
  // runs whose three passes all have batched forms step in the persistent kernel
#ifndef MWF_NO_PERSIST
  for (RunHost& r : h->runs) r.persist = r.d.precision == MWF_FP32 && r.xbf_nb && r.zb_lx && r.xbi_nb;
#endif
  // FP32 items by what their launch holds (a run's results do not depend on the width, bitwise).  One run, us a
  // step with the widest items, by the knobs, and with these: M4, MM = NN = 32 18.0 and 11.8, 64 22.5 and 16.3; M6,
  // 64 24.6 and 20.1.  Warp-line runs when the rule came in, and now: M4 36 40.5, 22.8 and 21.8, 72 54.2,
  // 28.9 and 27.7; M6 72 54.4, 39.1 and 33.8; eight M4 36 43.5, 32.9 and 32.1.  Full launches keep the widest.
  {
    std::map<std::vector<int>, std::vector<ItemWidth>> xf, z, xi, xwf, xwi, zw;
    for (RunHost& r : h->runs) {
      const mwf_run_desc& d = r.d;
      const int pset = r.persist ? 1 : 0;
      if (r.xbf_nb) xf[{pset, d.MM}].push_back({&r.xbf_nb, d.NN, d.K0, d.xf_cols != 0});
      if (r.xbi_nb) xi[{pset, d.MM}].push_back({&r.xbi_nb, d.NN, d.K0, d.xi_cols != 0});
      if (r.zb_lx) z[{pset, d.K0, d.NN}].push_back({&r.zb_lx, r.X, 1, d.z_lines != 0});
      if (r.xw_fnb) xwf[{r.xw_fnt}].push_back({&r.xw_fnb, d.NN, d.K0, false});
      if (r.xw_inb) xwi[{r.xw_int}].push_back({&r.xw_inb, d.NN, d.K0, false});
      if (r.zw_lines) zw[{d.K0, r.zw_ns, r.zw_nt}].push_back({&r.zw_lines, r.X, 1, false});
    }
    // rounds that the resident CTAs make; past these the narrower items' setup costs more (at
    // M4 128 x 128 modes and 228 x forward items 33.7 us, with 128 of them 30.0)
    for (auto& g : xf) spread_items(g.second, 152, false);
    for (auto& g : xi) spread_items(g.second, 304, false);
    for (auto& g : z) spread_items(g.second, 304, false);
    for (auto& g : xwf) spread_items(g.second, 304, true);
    for (auto& g : xwi) spread_items(g.second, 456, true);
    for (auto& g : zw) spread_items(g.second, 304, false);
  }
  // launch groups of the other runs and of the runs that can step in the persistent kernel
  auto build_groups = [&](bool pset) {
  for (int prec = 0; prec < 2; ++prec) {
    // subset-split FP32 x forward: one launch per MM; an item writes u_k, v_k, w_k of one
    // wall-normal mode k and their x derivatives for a block of columns
    for (int MM : kXbSizes) {
      Launch L{0, prec, 0, 0, kXbThreads, 0, items.size(), 0};
      L.xbMM = MM;
      for (int i = 0; i < n_runs; ++i) {
        const RunHost& r = h->runs[i];
        if (r.persist != pset || r.d.precision != prec || r.d.MM != MM || !r.xbf_nb) continue;
        for (int n0 = 0; n0 < r.d.NN; n0 += r.xbf_nb)
          for (int k = 0; k < r.d.K0; ++k) items.push_back(WorkItem{i, n0, k, 0});
        L.smem = std::max(L.smem, xbf_smem(MM, r.xbf_nb));
      }
      L.nitems = (int)(items.size() - L.item_off);
      if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
    }
    // x forward, grouped by block size
    for (int nt : {kXThreadsSmall, kXfThreads}) {
      Launch L{0, prec, 0, 0, nt, 0, items.size(), 0};
      for (int i = 0; i < n_runs; ++i) {
        const RunHost& r = h->runs[i];
        if (r.persist != pset || r.d.precision != prec || r.x_nt != nt || r.xbf_nb || r.xw_fnb || r.fx) continue;
        for (int n0 = 0; n0 < r.d.NN; n0 += r.xf_nb)
          for (int f = 0; f < 2 * r.KK; ++f) items.push_back(WorkItem{i, n0, f, 0});
        L.smem = std::max(L.smem, xpass_smem(prec, (size_t)r.xf_nb * r.X));
      }
      L.nitems = (int)(items.size() - L.item_off);
      if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
    }
    // batched FP32 z pass: one launch per (model, NN)
    for (int K0 : {4, 6})
      for (int Q : {32, 48, 64, 96, 128, 192, 256}) {
        Launch L{1, prec, K0, 0, kZbThreads, 0, items.size(), 0, Q};
        for (int i = 0; i < n_runs; ++i) {
          const RunHost& r = h->runs[i];
          if (r.persist != pset || r.d.precision != prec || r.d.K0 != K0 || r.d.NN != Q || !r.zb_lx) continue;
          for (int x0 = 0; x0 < r.X; x0 += r.zb_lx) items.push_back(WorkItem{i, x0, 0, 0});
          L.smem = std::max(L.smem, zb_smem(K0, Q, r.zb_lx));
        }
        L.nitems = (int)(items.size() - L.item_off);
        if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
      }
    for (int K0 : {4, 6})
      for (int ppt : {1, 2})
        for (int nt : {kZThreadsSmall, kZThreads}) {
        Launch L{1, prec, K0, ppt, nt, 0, items.size(), 0};
        for (int i = 0; i < n_runs; ++i) {
          const RunHost& r = h->runs[i];
          if (r.persist != pset || r.d.precision != prec || r.d.K0 != K0 || r.z_ppt != ppt || r.z_nt != nt || r.zb_lx || r.zw_lines || r.fx) continue;
          // FP32: one item per line block running the three z-subsets, summed (RunDesc::z_sum),
          // so the x-inverse pass reads one partial instead of three
          for (int x0 = 0; x0 < r.X; x0 += r.z_lx) {
            if (zpass_summed(prec)) items.push_back(WorkItem{i, x0, 3, 0});
            else
              for (int sub = 0; sub < 3; ++sub) items.push_back(WorkItem{i, x0, sub, 0});
          }
          L.smem = zpass_smem(prec, K0, ppt, nt);
        }
        L.nitems = (int)(items.size() - L.item_off);
        if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
      }
    for (int MM : kXbSizes) {
      Launch L{2, prec, 0, 0, kXbThreads, 0, items.size(), 0};
      L.xbMM = MM;
      for (int i = 0; i < n_runs; ++i) {
        const RunHost& r = h->runs[i];
        if (r.persist != pset || r.d.precision != prec || r.d.MM != MM || !r.xbi_nb) continue;
        for (int n0 = 0; n0 < r.d.NN; n0 += r.xbi_nb)
          for (int k = 0; k < r.d.K0; ++k) items.push_back(WorkItem{i, n0, k, 0});
        L.smem = std::max(L.smem, xbi_smem(MM, r.xbi_nb));
      }
      L.nitems = (int)(items.size() - L.item_off);
      if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
    }
    for (int nt : {kXThreadsSmall, kXiThreads}) {
      Launch L{2, prec, 0, 0, nt, 0, items.size(), 0};
      for (int i = 0; i < n_runs; ++i) {
        const RunHost& r = h->runs[i];
        if (r.persist != pset || r.d.precision != prec || r.x_nt != nt || r.xbi_nb || r.xw_inb || r.fx) continue;
        for (int n0 = 0; n0 < r.d.NN; n0 += r.xi_nb)
          for (int k = 0; k < r.d.K0; ++k) items.push_back(WorkItem{i, n0, k, 0});
        L.smem = std::max(L.smem, xpass_smem(prec, (size_t)3 * r.xi_nb * r.X));
      }
      L.nitems = (int)(items.size() - L.item_off);
      if (L.nitems) { L.persist_group = pset; h->launches.push_back(L); }
    }
  }
  };
  build_groups(false);
  build_groups(true);
  // FP32 x passes with a warp per line: one launch per pass and block size
  for (int kind : {0, 2})
    for (int nt : {256, 512}) {
      Launch L{kind, 1, 0, 0, nt, 0, items.size(), 0};
      L.xw = true;
      for (int i = 0; i < n_runs; ++i) {
        const RunHost& r = h->runs[i];
        if (!r.xw_fnb || (kind == 0 ? r.xw_fnt : r.xw_int) != nt) continue;
        const int nb = kind == 0 ? r.xw_fnb : r.xw_inb, LS = inplace_line(r.d.MM);
        for (int n0 = 0; n0 < r.d.NN; n0 += nb)
          for (int k = 0; k < r.d.K0; ++k) items.push_back(WorkItem{i, n0, k, 0});
        L.smem = std::max(L.smem, kind == 0 ? xw_fsmem(r.d.MM, LS, r.xw_nd, nb) : xw_ismem(r.d.MM, LS, nb));
      }
      L.nitems = (int)(items.size() - L.item_off);
      if (L.nitems) h->launches.push_back(L);
    }
  // FP32 z pass with a warp per line: one launch per model, subsets at once and block size
  for (int K0 : {4, 6})
    for (int ns : {3, 1})
      for (int nt : {256, 512, 576}) {
        Launch L{1, 1, K0, 0, nt, 0, items.size(), 0};
        L.zw_ns = ns;
        for (int i = 0; i < n_runs; ++i) {
          const RunHost& r = h->runs[i];
          if (!r.zw_lines || r.d.K0 != K0 || r.zw_ns != ns || r.zw_nt != nt) continue;
          for (int x0 = 0; x0 < r.X; x0 += r.zw_lines) items.push_back(WorkItem{i, x0, 0, 0});
          L.smem = std::max(L.smem, zw_smem(K0, r.d.NN, inplace_line(r.d.NN), ns, r.zw_lines));
        }
        L.nitems = (int)(items.size() - L.item_off);
        if (L.nitems) h->launches.push_back(L);
      }
  // FP64 runs in fixed point: one launch per pass and block size (and model, for the z pass)
  for (int kind = 0; kind < 3; ++kind)
    for (int K0 : {4, 6})
      for (int nt : {256, 512, 544}) {
        if (kind != 1 && K0 == 6) continue;
        Launch L{kind, 0, K0, 0, nt, 0, items.size(), 0};
        L.fx = true;
        for (int i = 0; i < n_runs; ++i) {
          const RunHost& r = h->runs[i];
          if (!r.fx) continue;
          if (kind == 0 && nt == 256) {
            for (int n0 = 0; n0 < r.d.NN; n0 += r.fx_nb)
              for (int f = 0; f < 2 * r.KK; ++f) items.push_back(WorkItem{i, n0, f, 0});
            L.smem = std::max(L.smem, fx_xf_smem(r.d.MM, r.fx_nb));
          } else if (kind == 1 && r.fx_z_nt == nt && r.d.K0 == K0) {
            for (int x0 = 0; x0 < r.X; x0 += r.fx_lines)
              for (int sub = 0; sub < 3; ++sub) items.push_back(WorkItem{i, x0, sub, 0});
            L.smem = std::max(L.smem, fx_z_smem(K0, r.d.NN, r.fx_lines, r.fx_tab));
          } else if (kind == 2 && r.fx_xi_nt == nt) {
            for (int n0 = 0; n0 < r.d.NN; n0 += r.fx_xi_nb)
              for (int k = 0; k < r.d.K0; ++k) items.push_back(WorkItem{i, n0, k, 0});
            L.smem = std::max(L.smem, fx_xi_smem(r.d.MM, r.fx_xi_nb));
          }
        }
        L.nitems = (int)(items.size() - L.item_off);
        if (L.nitems) h->launches.push_back(L);
      }
  // the persistent step's items: a three-stage pipeline over groups of runs whose x-transformed
  // fields total at most kGroupBytes (the x forward of group p beside the z pass of group p-1 and
  // the x inverse of group p-2, each stage's lists merged in proportion), so every item's
  // prerequisites hold lower tickets
  std::vector<PersistItem> pitems;
  {
    auto size_index = [](int v) {
      for (int k = 0; k < 7; ++k)
        if (kXbSizes[k] == v) return k;
      return 255;
    };
    const size_t kGroupBytes = (size_t)40 << 20;
    std::vector<std::vector<int>> groups;
    size_t acc = 0;
    for (int i = 0; i < n_runs; ++i) {
      const RunHost& r = h->runs[i];
      if (!r.persist) continue;
      const size_t tb = (size_t)2 * r.KK * r.X * r.d.NN * 8;
      if (groups.empty() || acc + tb > kGroupBytes) {
        groups.emplace_back();
        acc = 0;
      }
      groups.back().push_back(i);
      acc += tb;
    }
    auto stage_items = [&](int g, int pass) {
      std::vector<PersistItem> v;
      for (int i : groups[g]) {
        const RunHost& r = h->runs[i];
        if (pass == 0) {
          for (int n0 = 0; n0 < r.d.NN; n0 += r.xbf_nb)
            for (int k = 0; k < r.d.K0; ++k) v.push_back(PersistItem{i, n0, k, size_index(r.d.MM)});
        } else if (pass == 1) {
          const int kind = r.d.K0 == 4 ? 1 : 2;
          for (int x0 = 0; x0 < r.X; x0 += r.zb_lx) v.push_back(PersistItem{i, x0, 0, kind << 8 | size_index(r.d.NN)});
        } else {
          for (int n0 = 0; n0 < r.d.NN; n0 += r.xbi_nb)
            for (int k = 0; k < r.d.K0; ++k) v.push_back(PersistItem{i, n0, k, 3 << 8 | size_index(r.d.MM)});
        }
      }
      return v;
    };
    const int G = (int)groups.size();
    for (int p = 0; p < G + 2; ++p) {
      std::vector<std::vector<PersistItem>> lists;
      if (p < G) lists.push_back(stage_items(p, 0));
      if (p >= 1 && p - 1 < G) lists.push_back(stage_items(p - 1, 1));
      if (p >= 2 && p - 2 < G) lists.push_back(stage_items(p - 2, 2));
      struct Key { double key; int li, j; };
      std::vector<Key> keys;
      for (int li = 0; li < (int)lists.size(); ++li)
        for (int j = 0; j < (int)lists[li].size(); ++j) keys.push_back(Key{(j + 0.5) / lists[li].size(), li, j});
      std::stable_sort(keys.begin(), keys.end(), [](const Key& x, const Key& y) { return x.key < y.key; });
      for (const Key& k : keys) pitems.push_back(lists[k.li][k.j]);
    }
    for (const PersistItem& it : pitems)
      if ((it.code & 0xff) > 6) {
        free_handle(h);
        return fail(MWF_ERR_SIZE, "persistent step: no batched kernel for run %d", it.run);
      }
    for (const RunHost& r : h->runs)
      if (r.persist)
        h->persist_smem = std::max({h->persist_smem, zb_smem(r.d.K0, r.d.NN, r.zb_lx), xbf_smem(r.d.MM, r.xbf_nb),
                                    xbi_smem(r.d.MM, r.xbi_nb)});
  }
  // launch order: all x-forward, then z, then x-inverse (independent precisions interleave)
  std::stable_sort(h->launches.begin(), h->launches.end(),
                   [](const Launch& a, const Launch& b) { return a.kind < b.kind; });
  const size_t off_items = o; o = align_up(o + sizeof(WorkItem) * items.size(), 256);
  const size_t off_pitems = o; o = align_up(o + sizeof(PersistItem) * pitems.size(), 256);
  const size_t off_counters = o; o = align_up(o + sizeof(int) * (1 + 2 * (size_t)n_runs), 256);
  size_t max_diag = 0;
  for (const RunHost& r : h->runs) max_diag = std::max(max_diag, (size_t)(r.n_diag_xf + r.n_diag_z));
  const size_t off_diag = o; o = align_up(o + sizeof(WorkItem) * max_diag, 256);
  const size_t off_err = o; o = align_up(o + 3 * sizeof(int), 256);
  const size_t off_part = o; o = align_up(o + sizeof(double) * mwf_handle::kEnergyParts, 256);
  const size_t off_stage = o; o = align_up(o + sizeof(double) * 2 * h->stage_elems, 256);
  h->arena_bytes = o;
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
    free_handle(h);
    return fail(MWF_ERR_CUDA, "stream creation failed");
  }
  if (cudaHostAlloc(&h->h_out, sizeof(HostOut), cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    h->h_out = nullptr;
    free_handle(h);
    return fail(MWF_ERR_NOMEM, "cudaHostAlloc failed");
  }
  memset(h->h_out, 0, sizeof(HostOut));
  if (cudaMalloc(&h->arena, o) != cudaSuccess) {
    cudaGetLastError();
    h->arena = nullptr;
    free_handle(h);
    return fail(MWF_ERR_NOMEM, "cudaMalloc of %zu bytes failed", o);
  }
  h->d_runs = reinterpret_cast<RunDesc*>(h->arena + off_runs);
  h->d_items = reinterpret_cast<WorkItem*>(h->arena + off_items);
  h->d_diag_items = reinterpret_cast<WorkItem*>(h->arena + off_diag);
  h->d_err = reinterpret_cast<int*>(h->arena + off_err);
  h->d_flag = h->d_err + 1;
  h->d_partial = reinterpret_cast<double*>(h->arena + off_part);
  h->d_ticket = reinterpret_cast<unsigned*>(h->d_err + 2);
  h->d_stage = reinterpret_cast<double*>(h->arena + off_stage);
  h->d_pitems = h->arena + off_pitems;
  h->n_pitems = (int)pitems.size();
  h->d_counters = reinterpret_cast<int*>(h->arena + off_counters);
  h->counters_bytes = sizeof(int) * (1 + 2 * (size_t)n_runs);
  if (h->n_pitems) {
    h->persist_grid = persistent_grid(h->persist_smem);
    if (h->persist_grid <= 0) {
      free_handle(h);
      return fail(MWF_ERR_CUDA, "persistent step: the device holds no CTA with %zu bytes of shared memory",
                  h->persist_smem);
    }
  }
  int rc = MWF_OK;
  auto ck = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && rc == MWF_OK) rc = fail(MWF_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  };
  ck(cudaMemsetAsync(h->arena, 0, o, h->stream), "arena clear");
  // The uploads below are cudaMemcpy calls on the legacy default stream, which does not wait
  // for the handle's non-blocking stream: finish the clear first, or it can land after them
  // and zero the tables of the first runs.
  ck(cudaStreamSynchronize(h->stream), "arena clear");
  std::map<int, std::vector<long double>> root_tables;   // one per length, for all runs
  auto roots = [&](int N) -> const std::vector<long double>& {
    std::vector<long double>& v = root_tables[N];
    if (v.empty()) v = twiddles(N);
    return v;
  };
  std::vector<RunDesc> rds(n_runs);
  for (int i = 0; i < n_runs && rc == MWF_OK; ++i) {
    RunHost& r = h->runs[i];
    RunDesc& D = rds[i];
    memset(&D, 0, sizeof D);
    D.K0 = r.d.K0; D.MM = r.d.MM; D.NN = r.d.NN; D.M = r.M; D.X = r.X; D.Z = r.Z; D.K = r.K; D.KK = r.KK;
    D.prec = r.d.precision;
    D.xf_nb = r.xf_nb; D.xi_nb = r.xi_nb; D.z_lx = r.z_lx;
    D.z_sum = zpass_summed(r.d.precision == MWF_FP64 ? 0 : 1) ? 1 : 0;
    D.zb_lx = r.zb_lx;
    D.xbf_nb = r.xbf_nb;
    D.xbi_nb = r.xbi_nb;
    D.xbf_items = r.xbf_nb ? ((r.d.NN + r.xbf_nb - 1) / r.xbf_nb) * r.d.K0 : 0;
    D.zb_items = r.zb_lx ? (r.X + r.zb_lx - 1) / r.zb_lx : 0;
    D.alpha = r.d.alpha; D.gamma = r.d.gamma; D.dt = r.d.dt;
    D.alpha_f = (float)r.d.alpha; D.gamma_f = (float)r.d.gamma;
    D.cth = cos(r.d.theta); D.sth = sin(r.d.theta);
    D.scale = 1.0 / ((double)r.X * (double)r.Z);
    D.c = h->arena + r.off_c;
    D.onl = h->arena + r.off_onl;
    D.inv_lhs = reinterpret_cast<const double*>(h->arena + r.off_ilhs);
    D.rhs = reinterpret_cast<const double*>(h->arena + r.off_rhs);
    D.T = h->arena + r.off_T;
    D.NLT = h->arena + r.off_NLT;
    D.twX = h->arena + r.off_twX;
    D.twQ = h->arena + r.off_twQ;
    D.twZ = h->arena + r.off_twZ;
    D.nst = reinterpret_cast<int*>(h->arena + r.off_nst);
    D.active = 1;
    if (!make_plan(r.X, D.planX, r.x_radix) || !make_plan(r.d.NN, D.planQ, r.z_radix)) {
      rc = fail(MWF_ERR_SIZE, "run %d: no FFT plan", i);
      break;
    }
    std::vector<double> il, rh;
    lhsrhs(r.d, il, rh);
    if (r.d.precision == MWF_FP64) {
      ck(cudaMemcpy(h->arena + r.off_ilhs, il.data(), il.size() * 8, cudaMemcpyHostToDevice), "lhs upload");
      ck(cudaMemcpy(h->arena + r.off_rhs, rh.data(), rh.size() * 8, cudaMemcpyHostToDevice), "rhs upload");
    } else {
      // FP32 runs: c' = A c + B (3 nl - onl) with A = rhs/lhs as a float pair (hi, lo) in the
      // 1/lhs slot and B = (dt/2)/lhs in the rhs slot, all formed in FP64
      const size_t n = il.size();
      std::vector<float> a(2 * n), b(n);
      for (size_t j = 0; j < n; ++j) {
        const double A = rh[j] * il[j];
        a[j] = (float)A;
        a[n + j] = (float)(A - (double)a[j]);
        b[j] = (float)(r.d.dt / 2.0 * il[j]);
      }
      ck(cudaMemcpy(h->arena + r.off_ilhs, a.data(), a.size() * 4, cudaMemcpyHostToDevice), "table upload");
      ck(cudaMemcpy(h->arena + r.off_rhs, b.data(), b.size() * 4, cudaMemcpyHostToDevice), "table upload");
    }
    auto up = [&](size_t off, int N) {
      const std::vector<long double>& v = roots(N);
      if (r.d.precision == MWF_FP64) {
        const std::vector<double> t(v.begin(), v.end());
        ck(cudaMemcpy(h->arena + off, t.data(), t.size() * 8, cudaMemcpyHostToDevice), "twiddle upload");
      } else {
        const std::vector<float> t(v.begin(), v.end());
        ck(cudaMemcpy(h->arena + off, t.data(), t.size() * 4, cudaMemcpyHostToDevice), "twiddle upload");
      }
    };
    up(r.off_twX, r.X);
    up(r.off_twQ, r.d.NN);
    up(r.off_twZ, r.Z);
    // in-place FP32 transforms of length N, their stage twiddles at off
    auto inplace = [&](int N, FxPlan& pl, size_t off, std::vector<unsigned short>& rev) {
      const std::vector<long double>& v = roots(3 * N);
      std::vector<float2> w(3 * (size_t)N), t;
      for (size_t j = 0; j < w.size(); ++j) w[j] = make_float2((float)v[2 * j], (float)v[2 * j + 1]);
      if (!make_fx_plan(N, w, false, pl, t, rev) || t.size() > (size_t)N) {
        rc = fail(MWF_ERR_SIZE, "run %d: no in-place FFT plan", i);
        return;
      }
      if (!t.empty()) ck(cudaMemcpy(h->arena + off, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice), "twiddle upload");
    };
    std::vector<unsigned short> rev;
    if (r.zw_lines) {
      inplace(r.d.NN, D.zw_plan, r.off_zw, rev);
      D.zw_lines = r.zw_lines;
      D.zw_tw = reinterpret_cast<const float2*>(h->arena + r.off_zw);
    }
    if (r.xw_fnb) {
      const size_t off_rev = align_up(r.off_xw + sizeof(float2) * (size_t)r.d.MM, 256);
      inplace(r.d.MM, D.xw_plan, r.off_xw, rev);
      if (!rev.empty()) ck(cudaMemcpy(h->arena + off_rev, rev.data(), rev.size() * sizeof(unsigned short), cudaMemcpyHostToDevice), "order upload");
      D.xw_fnb = r.xw_fnb; D.xw_inb = r.xw_inb; D.xw_nd = r.xw_nd;
      D.xw_tw = reinterpret_cast<const float2*>(h->arena + r.off_xw);
      D.xw_rev = reinterpret_cast<const unsigned short*>(h->arena + off_rev);
    }
    if (rc != MWF_OK) break;
    if (r.fx) {
      const RunHost::FxOff fo = r.fx_off();
      std::vector<int4> gn(r.d.NN);
      FxTables t;
      if (!make_fx_tables(r.d.MM, r.d.NN, roots(r.X), roots(r.Z), D, t)) {
        rc = fail(MWF_ERR_SIZE, "run %d: no fixed-point FFT plan", i);
        break;
      }
      // mantissa in [1/2, 1) and exponent of gamma n and of the powers 0 .. 3 of alpha m
      auto factor = [](double v) {
        int ex = 0;
        const long long w = (long long)std::ldexp(std::frexp(v, &ex), 62);
        const int l = (int)(unsigned)w;
        return make_int4((int)((w - l) >> 32), l, ex, 0);
      };
      std::vector<int4> mp(4 * (size_t)r.d.MM);
      std::vector<double> ms(2 * (size_t)r.d.MM);
      for (int n = 0; n < r.d.NN; ++n) gn[n] = factor(r.d.gamma * n);
      for (int m = 0; m < r.d.MM; ++m) {
        const double m1 = r.d.alpha * m;
        double v = 1.0;
        for (int p = 0; p < 4; ++p, v *= m1) mp[(size_t)p * r.d.MM + m] = factor(v);
        ms[2 * (size_t)m] = m1 * D.scale;
        ms[2 * (size_t)m + 1] = m1 * m1 * D.scale;
      }
      auto put = [&](size_t off, const void* p, size_t bytes) {
        if (bytes) ck(cudaMemcpy(h->arena + off, p, bytes, cudaMemcpyHostToDevice), "fixed-point table upload");
      };
      put(fo.twX, t.wX.data(), t.wX.size() * sizeof(int4));
      put(fo.twZ, t.wZ.data(), t.wZ.size() * sizeof(int4));
      put(fo.twM, t.tM.data(), t.tM.size() * sizeof(int4));
      put(fo.twQ, t.tQ.data(), t.tQ.size() * sizeof(int4));
      put(fo.gn, gn.data(), gn.size() * sizeof(int4));
      put(fo.mp, mp.data(), mp.size() * sizeof(int4));
      put(fo.ms, ms.data(), ms.size() * 8);
      put(fo.rev, t.rev.data(), t.rev.size() * sizeof(unsigned short));
      put(fo.revQ, t.revQ.data(), t.revQ.size() * sizeof(unsigned short));
      D.fx = 1;
      D.fx_nb = r.fx_nb; D.fx_xi_nb = r.fx_xi_nb; D.fx_nblk = r.fx_nblk; D.fx_lines = r.fx_lines; D.fx_tab = r.fx_tab; D.fx_group = r.fx_group;
      D.fx_twX = reinterpret_cast<const int4*>(h->arena + fo.twX);
      D.fx_twZ = reinterpret_cast<const int4*>(h->arena + fo.twZ);
      D.fx_twM = reinterpret_cast<const int4*>(h->arena + fo.twM);
      D.fx_twQ = reinterpret_cast<const int4*>(h->arena + fo.twQ);
      D.fx_gn = reinterpret_cast<const int4*>(h->arena + fo.gn);
      D.fx_mp = reinterpret_cast<const int4*>(h->arena + fo.mp);
      D.fx_ms = reinterpret_cast<const double2*>(h->arena + fo.ms);
      D.fx_rev = reinterpret_cast<const unsigned short*>(h->arena + fo.rev);
      D.fx_revQ = reinterpret_cast<const unsigned short*>(h->arena + fo.revQ);
      D.fx_colE = reinterpret_cast<int*>(h->arena + fo.colE);
      D.fx_blkE = reinterpret_cast<int*>(h->arena + fo.blkE);
      D.fx_rowE = reinterpret_cast<int*>(h->arena + fo.rowE);
      D.fx_minE = reinterpret_cast<int*>(h->arena + fo.minE);
      D.fx_rowP = reinterpret_cast<unsigned*>(h->arena + fo.rowP);
    }
    const int one = 1;
    ck(cudaMemcpy(h->arena + r.off_nst, &one, sizeof(int), cudaMemcpyHostToDevice), "nst init");
  }
  if (rc == MWF_OK) {
    ck(cudaMemcpy(h->d_runs, rds.data(), sizeof(RunDesc) * n_runs, cudaMemcpyHostToDevice), "desc upload");
    ck(cudaMemcpy(h->d_items, items.data(), sizeof(WorkItem) * items.size(), cudaMemcpyHostToDevice), "item upload");
    if (!pitems.empty())
      ck(cudaMemcpy(h->d_pitems, pitems.data(), sizeof(PersistItem) * pitems.size(), cudaMemcpyHostToDevice),
         "persistent item upload");
    ck(cudaDeviceSynchronize(), "create sync");
  }
  if (rc == MWF_OK) rc = build_graph(h, 1, &h->graph1);
  if (rc == MWF_OK) rc = build_graph(h, mwf_handle::kGraphSteps, &h->graphG);
  if (rc != MWF_OK) { free_handle(h); return rc; }
  *out = h;
  return MWF_OK;
}

int mwf_destroy(mwf_handle* h) {
  if (!h) return fail(MWF_ERR_ARG, "mwf_destroy: null handle");
  cudaSetDevice(h->device);
  cudaStreamSynchronize(h->stream);
  free_handle(h);
  return MWF_OK;
}

static int check_run(mwf_handle* h, int run) {
  if (!h) return fail(MWF_ERR_ARG, "null handle");
  if (run < 0 || run >= (int)h->runs.size()) return fail(MWF_ERR_ARG, "run index %d out of range", run);
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  return MWF_OK;
}

// State copies between the caller's split arrays (reference layout) and array `off` of run r, queued
// on the handle's stream.  Pinned arrays are accessed by the conversion kernel itself, in place of
// two staging copies per direction and the copy of the error word: get_state of a 27 KB, 1.8 MB and
// 45 MB array pair took 21.8, 42.5 and 536 us with copies and takes 14.0, 33 and 493 us.
static int state_in(mwf_handle* h, const RunHost& r, size_t off, const double* re, const double* im) {
  const bool f64 = r.d.precision == MWF_FP64;
  cudaError_t e;
  if (device_reads_host(re, r.csz) && device_reads_host(im, r.csz)) {
    e = f64 ? launch_host_to_dev_f64(re, im, h->arena + off, r.K, r.M, r.d.NN, h->stream)
            : launch_host_to_dev_f32(re, im, h->arena + off, r.K, r.M, r.d.NN, h->stream);
  } else {
    double* sre = h->d_stage;
    double* sim = h->d_stage + h->stage_elems;
    CK(cudaMemcpyAsync(sre, re, r.csz * 8, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(sim, im, r.csz * 8, cudaMemcpyHostToDevice, h->stream));
    e = f64 ? launch_ref_to_dev_f64(sre, sim, h->arena + off, r.K, r.M, r.d.NN, h->stream)
            : launch_ref_to_dev_f32(sre, sim, h->arena + off, r.K, r.M, r.d.NN, h->stream);
  }
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "state conversion: %s", cudaGetErrorString(e));
  return MWF_OK;
}

// The error word follows into h_out (finish_call).
static int state_out(mwf_handle* h, const RunHost& r, size_t off, double* re, double* im) {
  const bool f64 = r.d.precision == MWF_FP64;
  const bool direct = device_reads_host(re, r.csz) && device_reads_host(im, r.csz);
  double* sre = direct ? re : h->d_stage;
  double* sim = direct ? im : h->d_stage + h->stage_elems;
  const cudaError_t e = f64 ? launch_dev_to_ref_f64(h->arena + off, sre, sim, r.K, r.M, r.d.NN, h->stream, h->d_err, h->h_out)
                            : launch_dev_to_ref_f32(h->arena + off, sre, sim, r.K, r.M, r.d.NN, h->stream, h->d_err, h->h_out);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "state conversion: %s", cudaGetErrorString(e));
  if (!direct) {
    CK(cudaMemcpyAsync(re, sre, r.csz * 8, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(im, sim, r.csz * 8, cudaMemcpyDeviceToHost, h->stream));
  }
  return MWF_OK;
}

int mwf_set_state(mwf_handle* h, int run, const double* re, const double* im) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!re || !im) return fail(MWF_ERR_ARG, "mwf_set_state: null state array");
  const RunHost& r = h->runs[run];
  rc = state_in(h, r, r.off_c, re, im);
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->stream));
  return MWF_OK;
}

int mwf_get_state(mwf_handle* h, int run, double* re, double* im) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!re || !im) return fail(MWF_ERR_ARG, "mwf_get_state: null state array");
  const RunHost& r = h->runs[run];
  rc = state_out(h, r, r.off_c, re, im);
  return rc ? rc : finish_call(h);
}

int mwf_get_history(mwf_handle* h, int run, double* re, double* im, int* euler_next) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!re || !im || !euler_next) return fail(MWF_ERR_ARG, "mwf_get_history: null argument");
  const RunHost& r = h->runs[run];
  rc = state_out(h, r, r.off_onl, re, im);
  if (rc) return rc;
  CK(cudaMemcpyAsync(euler_next, h->arena + r.off_nst, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  return finish_call(h);
}

int mwf_set_history(mwf_handle* h, int run, const double* re, const double* im, int euler_next) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!re || !im) return fail(MWF_ERR_ARG, "mwf_set_history: null argument");
  const RunHost& r = h->runs[run];
  rc = state_in(h, r, r.off_onl, re, im);
  if (rc) return rc;
  const int v = euler_next ? 1 : 0;
  if (v) h->euler_pending = true;
  CK(cudaMemcpyAsync(h->arena + r.off_nst, &v, sizeof(int), cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return MWF_OK;
}

int mwf_query(mwf_handle* h, int* idle) {
  if (!h || !idle) return fail(MWF_ERR_ARG, "mwf_query: null argument");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  const cudaError_t e = cudaStreamQuery(h->stream);
  if (e == cudaErrorNotReady) {
    *idle = 0;
    return MWF_OK;
  }
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_query: %s", cudaGetErrorString(e));
  *idle = 1;
  return MWF_OK;
}

int mwf_step_async(mwf_handle* h, int nsteps) {
  if (!h) return fail(MWF_ERR_ARG, "null handle");
  if (nsteps < 0) return fail(MWF_ERR_ARG, "nsteps < 0");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  int s = nsteps;
  if (s > 0 && h->euler_pending) {
    const int rc = enqueue_step(h, true);
    if (rc) return rc;
    h->euler_pending = false;
    --s;
  }
  while (s >= mwf_handle::kGraphSteps) {
    CK(cudaGraphLaunch(h->graphG, h->stream));
    s -= mwf_handle::kGraphSteps;
  }
  while (s-- > 0) CK(cudaGraphLaunch(h->graph1, h->stream));
  return MWF_OK;
}

int mwf_synchronize(mwf_handle* h) {
  if (!h) return fail(MWF_ERR_ARG, "null handle");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  return check_device_err(h);
}

int mwf_step(mwf_handle* h, int nsteps) {
  int rc = mwf_step_async(h, nsteps);
  if (rc) return rc;
  return mwf_synchronize(h);
}

int mwf_reset_history(mwf_handle* h, int run) {
  int rc = check_run(h, run);
  if (rc) return rc;
  const int one = 1;
  h->euler_pending = true;
  CK(cudaMemcpyAsync(h->arena + h->runs[run].off_nst, &one, sizeof(int), cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return MWF_OK;
}

int mwf_phys_diagnostics(mwf_handle* h, int run, double threshold, double* count_above, double* energy) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!count_above || !energy) return fail(MWF_ERR_ARG, "mwf_phys_diagnostics: null output");
  const RunHost& r = h->runs[run];
  if (!r.active) return fail(MWF_ERR_ARG, "run %d is not active", run);
  const int prec = r.d.precision;
  const bool fx = r.fx && fx_diag_fits(r.KK, r.d.NN);
  const int nz = fx ? r.X : r.n_diag_z;
  cudaStream_t st = h->stream;
  RunDesc* d = h->d_runs + run;
  cudaError_t e;
  if (fx) {
    e = launch_spec_x_backward_fx(h->d_runs, run, r.d.MM, r.KK, r.d.NN, nullptr, st);
    if (e == cudaSuccess)
      e = launch_diag_z_fx(h->d_runs, run, r.X, r.KK, r.d.NN, threshold, reinterpret_cast<double*>(h->arena + r.off_NLT), st);
  } else {
    rc = diag_x_forward(h, run, true, e);
    if (rc) return rc;
    CK(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(d) + offsetof(RunDesc, diag_ct), &threshold, sizeof(double),
                       cudaMemcpyHostToDevice, st));
    const size_t zsm = zpass_smem(prec, r.d.K0, r.z_ppt, r.z_nt);
    if (e == cudaSuccess)
      e = prec == MWF_FP64
              ? launch_z_diag_f64(r.d.K0, r.z_ppt, r.z_nt, h->d_runs, h->d_diag_items + r.n_diag_xf, r.n_diag_z, zsm, h->d_err, st)
              : launch_z_diag_f32(r.d.K0, r.z_ppt, r.z_nt, h->d_runs, h->d_diag_items + r.n_diag_xf, r.n_diag_z, zsm, h->d_err, st);
  }
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "diagnostic launch: %s", cudaGetErrorString(e));
  std::vector<double> part(2 * (size_t)nz);
  CK(cudaMemcpyAsync(part.data(), h->arena + r.off_NLT, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, st));
  rc = check_device_err(h);
  if (rc) return rc;
  double cnt = 0.0, sum = 0.0, comp = 0.0;
  for (int i = 0; i < nz; ++i) {
    cnt += part[2 * i];
    const double t = part[2 * i + 1];
    const double y = sum + t;
    comp += (fabs(sum) >= fabs(t)) ? (sum - y) + t : (t - y) + sum;
    sum = y;
  }
  *count_above = cnt;
  *energy = (sum + comp) / ((double)r.X * (double)r.Z);
  return MWF_OK;
}

int mwf_set_active(mwf_handle* h, int run, int active) {
  int rc = check_run(h, run);
  if (rc) return rc;
  const int v = active ? 1 : 0;
  h->runs[run].active = v;
  RunDesc* d = h->d_runs + run;
  CK(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(d) + offsetof(RunDesc, active), &v, sizeof(int),
                     cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return MWF_OK;
}

int mwf_test_copy_timeout(mwf_handle* h, int run, unsigned extra_bytes, double wait_ms) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!(wait_ms >= 0.0) || wait_ms > 1000.0 || extra_bytes % 16 || extra_bytes > (1u << 20))
    return fail(MWF_ERR_ARG, "mwf_test_copy_timeout: wait_ms must be in [0, 1000] and extra_bytes a multiple "
                             "of 16 up to 1 MiB");
  const unsigned long long ns = (unsigned long long)(wait_ms * 1e6);
  RunDesc* d = h->d_runs + run;
  CK(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(d) + offsetof(RunDesc, test_tx_extra), &extra_bytes,
                     sizeof(unsigned), cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(d) + offsetof(RunDesc, test_wait_ns), &ns,
                     sizeof(unsigned long long), cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return MWF_OK;
}

int mwf_energy(mwf_handle* h, int run, double* e) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!e) return fail(MWF_ERR_ARG, "mwf_energy: null output");
  const RunHost& r = h->runs[run];
  const size_t pts = (size_t)r.M * r.d.NN;
  const int parts = (int)std::min<size_t>(mwf_handle::kEnergyParts, (pts + kEnergyThreads - 1) / kEnergyThreads);
  const cudaError_t ce =
      r.d.precision == MWF_FP64
          ? launch_energy_f64(h->d_runs, run, h->d_partial, parts, h->d_flag, h->d_ticket, h->d_err, h->h_out, h->stream)
          : launch_energy_f32(h->d_runs, run, h->d_partial, parts, h->d_flag, h->d_ticket, h->d_err, h->h_out, h->stream);
  if (ce != cudaSuccess) return fail(MWF_ERR_CUDA, "energy launch: %s", cudaGetErrorString(ce));
  rc = finish_call(h);
  if (rc) return rc;
  const int flag = h->h_out->flag;
  *e = h->h_out->value;
  if (flag) return fail(MWF_ERR_NONFINITE, "run %d: state contains NaN/Inf", run);
  return MWF_OK;
}

// ---- state operations and diagnostics outside the timestep ----

int mwf_get_phys(mwf_handle* h, int run, double* p) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!p) return fail(MWF_ERR_ARG, "mwf_get_phys: null output");
  const RunHost& r = h->runs[run];
  if (!r.active) return fail(MWF_ERR_ARG, "run %d is not active", run);
  const int prec = r.d.precision;
  FftPlanDev pz{};
  if (!make_plan(r.Z, pz, prec == MWF_FP64 ? 12 : 16) || r.Z > kPhysVpt * kPhysThreads)
    return fail(MWF_ERR_SIZE, "no z plan for Z = %d", r.Z);
  cudaStream_t st = h->stream;
  const size_t zs = xpass_smem(prec, (size_t)r.Z);
  double* out = reinterpret_cast<double*>(h->arena + r.off_NLT);   // KK*X*Z doubles fit the NLT scratch
  cudaError_t e;
  if (r.fx) {
    e = launch_spec_x_backward_fx(h->d_runs, run, r.d.MM, r.KK, r.d.NN, nullptr, st);
    if (e == cudaSuccess) e = launch_phys_z_fx(h->d_runs, run, r.X, r.KK, r.d.NN, out, st);
  } else {
    rc = diag_x_forward(h, run, false, e);
    if (rc) return rc;
    if (e == cudaSuccess)
      e = prec == MWF_FP64 ? launch_phys_z_f64(h->d_runs, run, r.X, r.KK, pz, zs, out, h->d_err, st)
                           : launch_phys_z_f32(h->d_runs, run, r.X, r.KK, pz, zs, out, h->d_err, st);
  }
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "physical-field launch: %s", cudaGetErrorString(e));
  CK(cudaMemcpyAsync(p, out, sizeof(double) * (size_t)r.KK * r.X * r.Z, cudaMemcpyDeviceToHost, st));
  return check_device_err(h);
}

int mwf_spectrum_maxima(mwf_handle* h, int run, double* m_max, double* n_max) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!m_max || !n_max) return fail(MWF_ERR_ARG, "mwf_spectrum_maxima: null output");
  const RunHost& r = h->runs[run];
  const int MM = r.d.MM, NN = r.d.NN;
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(h->arena + r.off_NLT);
  cudaStream_t st = h->stream;
  CK(cudaMemsetAsync(mx, 0, sizeof(unsigned long long) * (MM + NN), st));
  cudaError_t e = r.d.precision == MWF_FP64 ? launch_spectrum_f64(h->d_runs, run, r.M, NN, mx, st)
                                            : launch_spectrum_f32(h->d_runs, run, r.M, NN, mx, st);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "spectrum launch: %s", cudaGetErrorString(e));
  std::vector<double> v(MM + NN);
  CK(cudaMemcpyAsync(v.data(), mx, sizeof(double) * v.size(), cudaMemcpyDeviceToHost, st));
  rc = check_device_err(h);
  if (rc) return rc;
  std::copy(v.begin(), v.begin() + MM, m_max);
  std::copy(v.begin() + MM, v.end(), n_max);
  return MWF_OK;
}

int mwf_history(mwf_handle* h, int run, double y, int n_probes, double* H) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!H) return fail(MWF_ERR_ARG, "mwf_history: null output");
  const RunHost& r = h->runs[run];
  if (n_probes < 1 || n_probes >= r.Z) return fail(MWF_ERR_ARG, "n_probes must be in [1, Z-1]");
  const int KK = r.KK, NN = r.d.NN, K0 = r.d.K0;
  std::vector<int> zs(n_probes);
  for (int j = 0; j < n_probes; ++j) zs[j] = (int)((long long)j * r.Z / n_probes) + 1;
  unsigned char* base = h->arena + r.off_NLT;
  double2* g = reinterpret_cast<double2*>(base);
  int* dz = reinterpret_cast<int*>(base + align_up(sizeof(double2) * (size_t)KK * NN, 256));
  double* dout = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(dz) + align_up(sizeof(int) * (size_t)n_probes, 256));
  cudaStream_t st = h->stream;
  CK(cudaMemcpyAsync(dz, zs.data(), sizeof(int) * zs.size(), cudaMemcpyHostToDevice, st));
  cudaError_t e = r.d.precision == MWF_FP64 ? launch_probes_f64(h->d_runs, run, K0, NN, g, dz, n_probes, dout, st)
                                            : launch_probes_f32(h->d_runs, run, K0, NN, g, dz, n_probes, dout, st);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "probe launch: %s", cudaGetErrorString(e));
  std::vector<double> V((size_t)n_probes * KK);
  CK(cudaMemcpyAsync(V.data(), dout, sizeof(double) * V.size(), cudaMemcpyDeviceToHost, st));
  rc = check_device_err(h);
  if (rc) return rc;
  // velU / velV / velW (modes.M4.f90:83-107, modes.M6.f90:81-111): u_k and w_k on 1,
  // sin(k beta y) (k odd), cos(k beta y) (k even); v_k on cos (k odd), sin (k even).
  const double beta = 0.5 * M_PI;
  std::vector<double> bu(K0), bv(K0);
  bu[0] = 1.0;
  for (int k = 1; k < K0; ++k) {
    bu[k] = (k & 1) ? std::sin(k * beta * y) : std::cos(k * beta * y);
    bv[k] = (k & 1) ? std::cos(k * beta * y) : std::sin(k * beta * y);
  }
  const double Lz = 2.0 * M_PI / r.d.gamma;
  for (int j = 0; j < n_probes; ++j) {
    const double* v = V.data() + (size_t)j * KK;
    double U = 0.0, Vv = 0.0, W = 0.0;
    for (int k = 0; k < K0; ++k) U += bu[k] * v[k];
    for (int k = 1; k < K0; ++k) Vv += bv[k] * v[K0 + k - 1];
    for (int k = 0; k < K0; ++k) W += bu[k] * v[2 * K0 - 1 + k];
    H[4 * j + 0] = zs[j] * Lz / r.Z;
    H[4 * j + 1] = U;
    H[4 * j + 2] = Vv;
    H[4 * j + 3] = W;
  }
  return MWF_OK;
}

static int set_nst(mwf_handle* h, const RunHost& r) {
  const int one = 1;
  h->euler_pending = true;
  CK(cudaMemcpyAsync(h->arena + r.off_nst, &one, sizeof(int), cudaMemcpyHostToDevice, h->stream));
  return MWF_OK;
}

int mwf_remap_x(mwf_handle* h, int run, int factor) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (factor < 1) return fail(MWF_ERR_ARG, "mwf_remap_x: factor must be >= 1");
  const RunHost& r = h->runs[run];
  const size_t cb = r.d.precision == MWF_FP64 ? 16 : 8;
  void* src = h->arena + r.off_T;          // the old state, in the transform scratch
  CK(cudaMemcpyAsync(src, h->arena + r.off_c, r.csz * cb, cudaMemcpyDeviceToDevice, h->stream));
  cudaError_t e = r.d.precision == MWF_FP64 ? launch_remap_x_f64(h->d_runs, run, src, r.csz, factor, h->stream)
                                            : launch_remap_x_f32(h->d_runs, run, src, r.csz, factor, h->stream);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "remap launch: %s", cudaGetErrorString(e));
  rc = set_nst(h, r);
  if (rc) return rc;
  return check_device_err(h);
}

int mwf_blend_state(mwf_handle* h, int run, int other, double d) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (other < 0 || other >= (int)h->runs.size()) return fail(MWF_ERR_ARG, "run index %d out of range", other);
  const RunHost& r = h->runs[run];
  const RunHost& o = h->runs[other];
  if (r.d.K0 != o.d.K0 || r.d.MM != o.d.MM || r.d.NN != o.d.NN || r.d.precision != o.d.precision)
    return fail(MWF_ERR_ARG, "mwf_blend_state: runs %d and %d differ in model, size or precision", run, other);
  if (!std::isfinite(d)) return fail(MWF_ERR_ARG, "mwf_blend_state: weight is not finite");
  cudaError_t e = r.d.precision == MWF_FP64 ? launch_blend_f64(h->d_runs, run, other, r.csz, d, h->stream)
                                            : launch_blend_f32(h->d_runs, run, other, r.csz, d, h->stream);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "blend launch: %s", cudaGetErrorString(e));
  rc = set_nst(h, r);
  if (rc) return rc;
  return check_device_err(h);
}

int mwf_add_noise(mwf_handle* h, int run, double scale, unsigned long long seed) {
  int rc = check_run(h, run);
  if (rc) return rc;
  if (!std::isfinite(scale)) return fail(MWF_ERR_ARG, "mwf_add_noise: scale is not finite");
  const RunHost& r = h->runs[run];
  cudaError_t e = r.d.precision == MWF_FP64 ? launch_noise_f64(h->d_runs, run, r.csz, scale, seed, h->stream)
                                            : launch_noise_f32(h->d_runs, run, r.csz, scale, seed, h->stream);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "noise launch: %s", cudaGetErrorString(e));
  return check_device_err(h);
}

// CUDA events (and a device buffer) released when the scope ends, on every return path of
// the timing helpers below, whose CK checks return early.
struct EventSet {
  std::vector<cudaEvent_t> ev;
  explicit EventSet(size_t n) : ev(n, nullptr) {}
  ~EventSet() {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
  }
  cudaError_t create() {
    for (cudaEvent_t& e : ev) {
      const cudaError_t r = cudaEventCreate(&e);
      if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
  }
  cudaEvent_t operator[](size_t i) const { return ev[i]; }
};
struct DeviceBuffer {
  void* p = nullptr;
  ~DeviceBuffer() {
    if (p) cudaFree(p);
  }
};

int mwf_step_timed(mwf_handle* h, int nsteps, double* ms) {
  if (!h || !ms) return fail(MWF_ERR_ARG, "mwf_step_timed: null argument");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  EventSet ev(2);
  CK(ev.create());
  CK(cudaEventRecord(ev[0], h->stream));
  int rc = mwf_step_async(h, nsteps);
  if (rc == MWF_OK) {
    CK(cudaEventRecord(ev[1], h->stream));
    CK(cudaEventSynchronize(ev[1]));
    float f = 0.f;
    CK(cudaEventElapsedTime(&f, ev[0], ev[1]));
    *ms = f;
    rc = check_device_err(h);
  }
  return rc;
}

int mwf_profile_passes(mwf_handle* h, int nreps, double* ms_per_pass) {
  if (!h || !ms_per_pass || nreps <= 0) return fail(MWF_ERR_ARG, "mwf_profile_passes: bad argument");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  const size_t nl = h->launches.size();
  EventSet ev(2 * nl * nreps);
  CK(ev.create());
  // the passes of one step, launched individually (the same launches the graph holds)
  int rc = MWF_OK;
  for (int rep = 0; rep < nreps && rc == MWF_OK; ++rep) {
    for (size_t i = 0; i < nl && rc == MWF_OK; ++i) {
      const Launch& L = h->launches[i];
      cudaStream_t st = h->stream;
      CK(cudaEventRecord(ev[2 * (rep * nl + i)], st));
      cudaError_t e = launch_pass(L, h->d_runs, h->d_items + L.item_off, h->d_err, st);
      if (e != cudaSuccess) rc = fail(MWF_ERR_CUDA, "profile launch: %s", cudaGetErrorString(e));
      CK(cudaEventRecord(ev[2 * (rep * nl + i) + 1], st));
    }
    CK(cudaMemsetAsync(h->arena + h->off_nst_all, 0, sizeof(int) * h->runs.size(), h->stream));
  }
  h->euler_pending = false;
  if (rc == MWF_OK) {
    CK(cudaStreamSynchronize(h->stream));
    double acc[3] = {0, 0, 0};
    for (int rep = 0; rep < nreps; ++rep)
      for (size_t i = 0; i < nl; ++i) {
        float f = 0.f;
        CK(cudaEventElapsedTime(&f, ev[2 * (rep * nl + i)], ev[2 * (rep * nl + i) + 1]));
        acc[h->launches[i].kind] += f;
      }
    for (int k = 0; k < 3; ++k) ms_per_pass[k] = acc[k] / nreps;
    rc = check_device_err(h);
  }
  return rc;
}

}  // extern "C"

namespace {

// Device memory of one stand-alone transform call (mwf_spec2phys / mwf_phys2spec), released on
// every return path: descriptor, error word, twiddles of X and Z, the spectral fields in the
// device layout, the x-transformed fields, the physical fields and the staging of the split
// Re/Im arrays, in one allocation.
struct TransformCall {
  unsigned char* mem = nullptr;
  RunHost r;
  RunDesc* d = nullptr;
  int* err = nullptr;
  double2* sp = nullptr;
  double* ph = nullptr;
  double* s_re = nullptr;
  double* s_im = nullptr;
  FftPlanDev pz{};
  size_t nspec = 0, nphys = 0;
  ~TransformCall() {
    if (mem) cudaFree(mem);
  }
};

int transform_setup(const mwf_run_desc* desc, const char* who, TransformCall& tc) {
  if (!desc) return fail(MWF_ERR_ARG, "%s: null argument", who);
  tc.r.d = *desc;
  tc.r.d.precision = MWF_FP64;
  tc.r.d.xf_cols = tc.r.d.xi_cols = tc.r.d.z_lines = tc.r.d.x_radix = tc.r.d.z_radix = 0;
  const char* why = "";
  if (!plan_run(tc.r, why)) return fail(MWF_ERR_SIZE, "%s: %s", who, why);
  RunHost& r = tc.r;
  if (r.Z > kPhysVpt * kPhysThreads) return fail(MWF_ERR_SIZE, "%s: 3NN = %d exceeds %d", who, r.Z, kPhysVpt * kPhysThreads);
  RunDesc D;
  memset(&D, 0, sizeof D);
  if (!make_plan(r.Z, tc.pz, 12) || !make_plan(r.X, D.planX, 12)) return fail(MWF_ERR_SIZE, "%s: no FFT plan", who);
  tc.nspec = (size_t)r.KK * r.M * r.d.NN;
  tc.nphys = (size_t)r.KK * r.Z * r.X;
  // descriptor, error word and tables first: one upload
  const std::vector<long double> lx = twiddles(r.X), lz = twiddles(r.Z);
  FxTables t;
  std::vector<double> twx, twz;
  if (!r.fx) {
    twx.assign(lx.begin(), lx.end());
    twz.assign(lz.begin(), lz.end());
  } else if (!make_fx_tables(r.d.MM, r.d.NN, lx, lz, D, t)) {
    return fail(MWF_ERR_SIZE, "%s: no fixed-point FFT plan", who);
  }
  std::vector<unsigned char> head(align_up(sizeof(RunDesc), 256) + 256);
  auto table = [&](const void* p, size_t bytes) {
    const size_t at = head.size();
    head.resize(align_up(at + bytes, 256));
    if (bytes) memcpy(head.data() + at, p, bytes);
    return at;
  };
  const size_t off_err = align_up(sizeof(RunDesc), 256);
  const size_t off_twX = r.fx ? table(t.wX.data(), t.wX.size() * sizeof(int4)) : table(twx.data(), twx.size() * 8);
  const size_t off_twZ = r.fx ? table(t.wZ.data(), t.wZ.size() * sizeof(int4)) : table(twz.data(), twz.size() * 8);
  const size_t off_tM = table(t.tM.data(), t.tM.size() * sizeof(int4)), off_tQ = table(t.tQ.data(), t.tQ.size() * sizeof(int4));
  const size_t off_rev = table(t.rev.data(), t.rev.size() * 2), off_revQ = table(t.revQ.data(), t.revQ.size() * 2);
  size_t o = head.size();
  const size_t off_sp = o; o = align_up(o + 16 * tc.nspec, 256);
  const size_t off_W = o; o = align_up(o + 16 * (size_t)r.KK * r.X * r.d.NN, 256);
  const size_t off_ph = o; o = align_up(o + 8 * tc.nphys, 256);
  const size_t off_re = o; o = align_up(o + 8 * tc.nspec, 256);
  const size_t off_im = o; o = align_up(o + 8 * tc.nspec, 256);
  if (cudaMalloc(&tc.mem, o) != cudaSuccess) {
    cudaGetLastError();
    tc.mem = nullptr;
    return fail(MWF_ERR_NOMEM, "%s: cudaMalloc of %zu bytes failed", who, o);
  }
  tc.d = reinterpret_cast<RunDesc*>(tc.mem);
  tc.err = reinterpret_cast<int*>(tc.mem + off_err);
  tc.sp = reinterpret_cast<double2*>(tc.mem + off_sp);
  tc.ph = reinterpret_cast<double*>(tc.mem + off_ph);
  tc.s_re = reinterpret_cast<double*>(tc.mem + off_re);
  tc.s_im = reinterpret_cast<double*>(tc.mem + off_im);
  D.K0 = r.d.K0; D.MM = r.d.MM; D.NN = r.d.NN; D.M = r.M; D.X = r.X; D.Z = r.Z; D.K = r.K; D.KK = r.KK;
  D.prec = 0;
  D.alpha = r.d.alpha; D.gamma = r.d.gamma; D.dt = r.d.dt;
  D.scale = 1.0 / ((double)r.X * (double)r.Z);
  D.T = tc.mem + off_W;
  D.twX = tc.mem + off_twX;
  D.twZ = tc.mem + off_twZ;
  D.fx_twX = reinterpret_cast<const int4*>(tc.mem + off_twX);
  D.fx_twZ = reinterpret_cast<const int4*>(tc.mem + off_twZ);
  D.fx_twM = reinterpret_cast<const int4*>(tc.mem + off_tM);
  D.fx_twQ = reinterpret_cast<const int4*>(tc.mem + off_tQ);
  D.fx_rev = reinterpret_cast<const unsigned short*>(tc.mem + off_rev);
  D.fx_revQ = reinterpret_cast<const unsigned short*>(tc.mem + off_revQ);
  D.active = 1;
  memcpy(head.data(), &D, sizeof D);
  CK(cudaMemcpy(tc.mem, head.data(), head.size(), cudaMemcpyHostToDevice));
  return MWF_OK;
}

int transform_finish(TransformCall& tc, const char* who) {
  int herr = 0;
  CK(cudaMemcpy(&herr, tc.err, sizeof(int), cudaMemcpyDeviceToHost));
  if (herr) return fail(MWF_ERR_DEVICE, "%s: kernel reported internal error flags 0x%x", who, herr);
  return MWF_OK;
}

}  // namespace

extern "C" {

int mwf_spec2phys(const mwf_run_desc* d, const double* s_re, const double* s_im, double* p) {
  if (!s_re || !s_im || !p) return fail(MWF_ERR_ARG, "mwf_spec2phys: null argument");
  TransformCall tc;
  int rc = transform_setup(d, "mwf_spec2phys", tc);
  if (rc) return rc;
  const RunHost& r = tc.r;
  CK(cudaMemcpy(tc.s_re, s_re, 8 * tc.nspec, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(tc.s_im, s_im, 8 * tc.nspec, cudaMemcpyHostToDevice));
  cudaError_t e = launch_ref_to_dev_f64(tc.s_re, tc.s_im, tc.sp, r.KK, r.M, r.d.NN, 0);
  if (e == cudaSuccess)
    e = r.fx ? launch_spec_x_backward_fx(tc.d, 0, r.d.MM, r.KK, r.d.NN, tc.sp, 0)
             : launch_spec_x_backward_f64(tc.d, 0, r.X, r.KK, r.d.NN, tc.sp, tc.err, 0);
  if (e == cudaSuccess)
    e = r.fx ? launch_phys_z_fx(tc.d, 0, r.X, r.KK, r.d.NN, tc.ph, 0)
             : launch_phys_z_f64(tc.d, 0, r.X, r.KK, tc.pz, xpass_smem(0, (size_t)r.Z), tc.ph, tc.err, 0);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_spec2phys: launch: %s", cudaGetErrorString(e));
  rc = transform_finish(tc, "mwf_spec2phys");
  if (rc) return rc;
  CK(cudaMemcpy(p, tc.ph, 8 * tc.nphys, cudaMemcpyDeviceToHost));
  return MWF_OK;
}

int mwf_phys2spec(const mwf_run_desc* d, const double* p, double* s_re, double* s_im) {
  if (!s_re || !s_im || !p) return fail(MWF_ERR_ARG, "mwf_phys2spec: null argument");
  TransformCall tc;
  int rc = transform_setup(d, "mwf_phys2spec", tc);
  if (rc) return rc;
  const RunHost& r = tc.r;
  CK(cudaMemcpy(tc.ph, p, 8 * tc.nphys, cudaMemcpyHostToDevice));
  cudaError_t e = r.fx ? launch_phys_z_forward_fx(tc.d, 0, r.X, r.KK, r.d.NN, tc.ph, 0)
                       : launch_phys_z_forward_f64(tc.d, 0, r.X, r.KK, r.Z, tc.pz, tc.ph, tc.err, 0);
  if (e == cudaSuccess)
    e = r.fx ? launch_spec_x_forward_fx(tc.d, 0, r.d.MM, r.KK, r.d.NN, tc.sp, 0)
             : launch_spec_x_forward_f64(tc.d, 0, r.X, r.KK, r.d.NN, tc.sp, tc.err, 0);
  if (e == cudaSuccess) e = launch_dev_to_ref_f64(tc.sp, tc.s_re, tc.s_im, r.KK, r.M, r.d.NN, 0);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_phys2spec: launch: %s", cudaGetErrorString(e));
  rc = transform_finish(tc, "mwf_phys2spec");
  if (rc) return rc;
  CK(cudaMemcpy(s_re, tc.s_re, 8 * tc.nspec, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(s_im, tc.s_im, 8 * tc.nspec, cudaMemcpyDeviceToHost));
  return MWF_OK;
}

int mwf_set_persistent(mwf_handle* h, int on) {
  if (!h) return fail(MWF_ERR_ARG, "mwf_set_persistent: null handle");
  if (cudaSetDevice(h->device) != cudaSuccess) return fail(MWF_ERR_CUDA, "cudaSetDevice failed");
  const bool want = on != 0;
  if (want == h->persist_mode) return MWF_OK;
  CK(cudaStreamSynchronize(h->stream));
  h->persist_mode = want;
  cudaGraphExec_t g1 = nullptr, gG = nullptr;
  int rc = build_graph(h, 1, &g1);
  if (rc == MWF_OK) rc = build_graph(h, mwf_handle::kGraphSteps, &gG);
  if (rc != MWF_OK) {
    if (g1) cudaGraphExecDestroy(g1);
    h->persist_mode = !want;
    return rc;
  }
  cudaGraphExecDestroy(h->graph1);
  cudaGraphExecDestroy(h->graphG);
  h->graph1 = g1;
  h->graphG = gG;
  return MWF_OK;
}

int mwf_kernels_per_step(mwf_handle* h, int* n) {
  if (!h || !n) return fail(MWF_ERR_ARG, "mwf_kernels_per_step: null argument");
  const bool persist = h->persist_mode && h->n_pitems;
  int k = persist ? 1 : 0;
  for (const Launch& L : h->launches) k += (persist && L.persist_group) ? 0 : 1;
  for (const RunHost& r : h->runs) k += (r.d.reflect ? 1 : 0) + (r.d.uvreflect ? 1 : 0) + (r.d.wreflect ? 1 : 0);
  *n = k;
  return MWF_OK;
}

int mwf_measure_fma_peak(int device, int which, double* tflops) {
  if (!tflops || (which != 0 && which != 1)) return fail(MWF_ERR_ARG, "mwf_measure_fma_peak: bad argument");
  CK(cudaSetDevice(device));
  int sms = 0;
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  DeviceBuffer out;
  const int blocks = sms * 8, threads = 256;
  CK(cudaMalloc(&out.p, (size_t)blocks * threads * 8));
  EventSet ev(2);
  CK(ev.create());
  const int iters = which == 0 ? 4096 : 65536;
  double best = 0.0;
  for (int rep = 0; rep < 4; ++rep) {
    CK(cudaEventRecord(ev[0], 0));
    cudaError_t e = launch_fma_probe(which, blocks, threads, iters, out.p, 0);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "fma probe: %s", cudaGetErrorString(e));
    CK(cudaEventRecord(ev[1], 0));
    CK(cudaEventSynchronize(ev[1]));
    float f = 0.f;
    CK(cudaEventElapsedTime(&f, ev[0], ev[1]));
    const double flops = 2.0 * kFmaChains * (double)iters * blocks * threads;
    if (rep > 0) best = std::max(best, flops / (f * 1e-3) / 1e12);
  }
  *tflops = best;
  return MWF_OK;
}

int mwf_host_alloc(size_t bytes, void** p) {
  if (!p) return fail(MWF_ERR_ARG, "mwf_host_alloc: null output");
  CK(cudaHostAlloc(p, bytes, cudaHostAllocDefault));
  return MWF_OK;
}

int mwf_host_free(void* p) {
  if (p) CK(cudaFreeHost(p));
  return MWF_OK;
}

int mwf_last_error(char* buf, size_t len) {
  if (buf && len) {
    strncpy(buf, g_err, len - 1);
    buf[len - 1] = 0;
  }
  return (int)strlen(g_err);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Time step for callers that cannot allocate device memory.
//
// Some callers of this library run where cudaMalloc is not theirs to call: a Fortran or
// C host code that owns every device buffer itself (CUDA Fortran or OpenACC device
// arrays, a memory pool it manages), or one that is not allowed to grow its device
// footprint after start-up.  mwf_step_noalloc advances a state that such a caller keeps
// in its own device arrays, with every intermediate array (device-layout state, FP64
// tables, twiddles, transposes) in the fixed file-scope array below instead of in memory
// the library allocates.  Every GPU that loads this module holds the array until the
// process exits; runs whose intermediates do not fit it are rejected.
// ---------------------------------------------------------------------------------------
#define MWF_NOALLOC_SCRATCH_BYTES ((size_t)64 << 20)

static __device__ __align__(256) unsigned char g_noalloc_scratch[MWF_NOALLOC_SCRATCH_BYTES];

namespace {

// var_LHSRHS (variables.f90:565-597) for one run, in the device layout [n][slot][m], with
// the reference's loop-order result per slot (slot < K0: psi_slot, else phi_{slot-K0+1})
// and the same FP64 operation order as the host tables (no contraction).  The stored form
// is the one the run's x-inverse pass reads, as mwf_create builds it: FP64 runs get 1/lhs
// and rhs as doubles; FP32 runs get A = rhs/lhs as a float pair (hi at ilhs[0..n), lo at
// ilhs[n..2n) as floats) and B = (dt/2)/lhs as floats in the rhs slot, formed in FP64.
__global__ void noalloc_tables_kernel(const RunDesc* rd, double Re, double drag, double vdrag, double hypo,
                                      int dragall, double* ilhs, double* rhs) {
  const int K0 = rd->K0, K = rd->K, M = rd->M, MM = rd->MM, NN = rd->NN;
  const double alpha = rd->alpha, gamma = rd->gamma, dt = rd->dt;
  const double beta = 3.1415926535897931 / 2.0;
  const size_t tot = (size_t)K * M * NN;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int ms = (int)(e % M);
    const int slot = (int)((e / M) % K);
    const int n = (int)(e / ((size_t)M * K));
    const int ma = ms < MM ? ms : M - ms;
    const double m2 = __dmul_rn(__dmul_rn(__dmul_rn(-alpha, (double)ma), alpha), (double)ma);
    const double n2 = __dmul_rn(__dmul_rn(__dmul_rn(-gamma, (double)n), gamma), (double)n);
    const bool psi = slot < K0;
    const int k = psi ? slot : slot - K0 + 1;
    const double k2 = __dmul_rn(__dmul_rn((double)(-k * k), beta), beta);
    const double lap = __dadd_rn(__dadd_rn(m2, k2), n2);
    const double hlap = __dadd_rn(m2, n2);
    const double ilap16 = hypo / lap;
    double inner = __dadd_rn(lap / Re, ilap16);
    if (dragall || k == 0) inner = __dsub_rn(inner, drag);
    const double tvl = __dsub_rn(1.0, __dmul_rn(dt, inner));
    double l, r;
    if (ms == 0 && n == 0) {
      if (slot == 0) { l = 1.0; r = 0.0; }
      else { l = tvl; r = 1.0; }
    } else if (psi) {
      l = __dmul_rn(tvl, hlap);
      r = hlap;
    } else {
      l = __dmul_rn(__dmul_rn(tvl, hlap), lap);
      if (dragall) l = __dadd_rn(l, __dmul_rn(__dmul_rn(__dmul_rn(dt, __dsub_rn(vdrag, drag)), hlap), hlap));
      r = __dmul_rn(hlap, lap);
    }
    const double il = 1.0 / l;
    if (rd->prec == MWF_FP64) {
      ilhs[e] = il;
      rhs[e] = r;
    } else {
      const double A = __dmul_rn(r, il);
      const float hi = __double2float_rn(A);
      float* a = reinterpret_cast<float*>(ilhs);
      a[e] = hi;
      a[tot + e] = __double2float_rn(__dsub_rn(A, (double)hi));
      reinterpret_cast<float*>(rhs)[e] = __double2float_rn(__dmul_rn(dt / 2.0, il));
    }
  }
}

}  // namespace

extern "C" int mwf_step_noalloc(const mwf_run_desc* d, double* c_re, double* c_im, double* onl_re,
                                double* onl_im, int first_step, int nsteps) {
  if (!d || !c_re || !c_im || !onl_re || !onl_im) return fail(MWF_ERR_ARG, "mwf_step_noalloc: null argument");
  if (nsteps < 0) return fail(MWF_ERR_ARG, "mwf_step_noalloc: nsteps < 0");
  if (d->reflect || d->uvreflect || d->wreflect)
    return fail(MWF_ERR_ARG, "mwf_step_noalloc: symmetry masks are not supported by this entry point");
  if (!(d->dt > 0) || !(d->Re > 0)) return fail(MWF_ERR_ARG, "mwf_step_noalloc: dt and Re must be > 0");
  RunHost r;
  r.d = *d;
  const char* why = "";
  if (!plan_run(r, why)) return fail(MWF_ERR_SIZE, "mwf_step_noalloc: %s", why);
  r.fx = false;                // the kernels below need no more than run_bytes' basic arrays
  r.zw_lines = r.xw_fnb = 0;
  const int prec = d->precision;
  const size_t cb = prec == MWF_FP64 ? 16 : 8;
  // work items of the three passes
  const int n_xf = ((d->NN + r.xf_nb - 1) / r.xf_nb) * 2 * r.KK;
  const int n_z = ((r.X + r.z_lx - 1) / r.z_lx) * 3;
  const int n_xi = ((d->NN + r.xi_nb - 1) / r.xi_nb) * d->K0;
  const int n_items = n_xf + n_z + n_xi;
  // scratch layout: descriptor | error word | items | run arrays
  const size_t off_desc = 0;
  const size_t off_err = align_up(sizeof(RunDesc), 256);
  const size_t off_items = off_err + 256;
  const size_t base = align_up(off_items + sizeof(WorkItem) * (size_t)n_items, 256);
  const size_t need = run_bytes(r, base);
  if (need > MWF_NOALLOC_SCRATCH_BYTES)
    return fail(MWF_ERR_SIZE,
                "mwf_step_noalloc: this run needs %zu bytes of intermediates; the entry point's fixed "
                "scratch holds %zu bytes (use mwf_create/mwf_step for larger runs)",
                need, (size_t)MWF_NOALLOC_SCRATCH_BYTES);
  // The array's name in host code is a host-side stand-in, not a device address: look up its
  // address on the current device at every call (cheap next to the uploads below, and never
  // stale after a device reset or a new primary context).
  unsigned char* sc = nullptr;
  {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr)
      return fail(MWF_ERR_CUDA, "mwf_step_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    sc = static_cast<unsigned char*>(ptr);
  }
  cudaStream_t st = 0;
  // descriptor
  RunDesc D;
  memset(&D, 0, sizeof D);
  D.K0 = d->K0; D.MM = d->MM; D.NN = d->NN; D.M = r.M; D.X = r.X; D.Z = r.Z; D.K = r.K; D.KK = r.KK;
  D.prec = prec;
  D.xf_nb = r.xf_nb; D.xi_nb = r.xi_nb; D.z_lx = r.z_lx;
  D.alpha = d->alpha; D.gamma = d->gamma; D.dt = d->dt;
  D.alpha_f = (float)d->alpha; D.gamma_f = (float)d->gamma;
  D.cth = cos(d->theta); D.sth = sin(d->theta);
  D.scale = 1.0 / ((double)r.X * (double)r.Z);
  D.c = sc + r.off_c;
  D.onl = sc + r.off_onl;
  D.inv_lhs = reinterpret_cast<const double*>(sc + r.off_ilhs);
  D.rhs = reinterpret_cast<const double*>(sc + r.off_rhs);
  D.T = sc + r.off_T;
  D.NLT = sc + r.off_NLT;
  D.twX = sc + r.off_twX;
  D.twQ = sc + r.off_twQ;
  D.twZ = sc + r.off_twZ;
  D.nst = reinterpret_cast<int*>(sc + r.off_nst);
  D.active = 1;
  if (!make_plan(r.X, D.planX, r.x_radix) || !make_plan(d->NN, D.planQ, r.z_radix))
    return fail(MWF_ERR_SIZE, "mwf_step_noalloc: no FFT plan");
  CK(cudaMemcpy(sc + off_desc, &D, sizeof D, cudaMemcpyHostToDevice));
  CK(cudaMemset(sc + off_err, 0, sizeof(int)));
  // work items, staged through a small stack buffer
  {
    WorkItem chunk[256];
    int nc = 0, done = 0;
    auto push = [&](WorkItem w) -> cudaError_t {
      chunk[nc++] = w;
      if (nc == 256) {
        cudaError_t e = cudaMemcpy(sc + off_items + sizeof(WorkItem) * done, chunk, sizeof chunk, cudaMemcpyHostToDevice);
        done += nc;
        nc = 0;
        return e;
      }
      return cudaSuccess;
    };
    for (int n0 = 0; n0 < d->NN; n0 += r.xf_nb)
      for (int f = 0; f < 2 * r.KK; ++f) CK(push(WorkItem{0, n0, f, 0}));
    for (int x0 = 0; x0 < r.X; x0 += r.z_lx)
      for (int sub = 0; sub < 3; ++sub) CK(push(WorkItem{0, x0, sub, 0}));
    for (int n0 = 0; n0 < d->NN; n0 += r.xi_nb)
      for (int k = 0; k < d->K0; ++k) CK(push(WorkItem{0, n0, k, 0}));
    if (nc) CK(cudaMemcpy(sc + off_items + sizeof(WorkItem) * done, chunk, sizeof(WorkItem) * nc, cudaMemcpyHostToDevice));
  }
  // twiddles, staged through a small stack buffer
  {
    double tw[2 * 256];
    float twf[2 * 256];
    const size_t offs[3] = {r.off_twX, r.off_twQ, r.off_twZ};
    const int lens[3] = {r.X, d->NN, r.Z};
    for (int q = 0; q < 3; ++q)
      for (int t0 = 0; t0 < lens[q]; t0 += 256) {
        const int cnt = std::min(256, lens[q] - t0);
        if (prec == MWF_FP64) {
          twiddles_into<double>(lens[q], t0, cnt, tw);
          CK(cudaMemcpy(sc + offs[q] + (size_t)t0 * cb, tw, (size_t)cnt * cb, cudaMemcpyHostToDevice));
        } else {
          twiddles_into<float>(lens[q], t0, cnt, twf);
          CK(cudaMemcpy(sc + offs[q] + (size_t)t0 * cb, twf, (size_t)cnt * cb, cudaMemcpyHostToDevice));
        }
      }
  }
  const RunDesc* d_desc = reinterpret_cast<const RunDesc*>(sc + off_desc);
  int* d_err = reinterpret_cast<int*>(sc + off_err);
  const WorkItem* d_items = reinterpret_cast<const WorkItem*>(sc + off_items);
  double* ilhs = reinterpret_cast<double*>(sc + r.off_ilhs);
  double* rhs = reinterpret_cast<double*>(sc + r.off_rhs);
  noalloc_tables_kernel<<<152 * 4, 256, 0, st>>>(d_desc, d->Re, d->drag, d->vdrag, d->hypo, d->dragall, ilhs, rhs);
  CK(cudaGetLastError());
  // caller state (reference layout, FP64) -> device layout in the scratch
  cudaError_t e;
  e = prec == MWF_FP64 ? launch_ref_to_dev_f64(c_re, c_im, sc + r.off_c, r.K, r.M, d->NN, st)
                       : launch_ref_to_dev_f32(c_re, c_im, sc + r.off_c, r.K, r.M, d->NN, st);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_step_noalloc: state conversion: %s", cudaGetErrorString(e));
  if (!first_step) {
    e = prec == MWF_FP64 ? launch_ref_to_dev_f64(onl_re, onl_im, sc + r.off_onl, r.K, r.M, d->NN, st)
                         : launch_ref_to_dev_f32(onl_re, onl_im, sc + r.off_onl, r.K, r.M, d->NN, st);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_step_noalloc: history conversion: %s", cudaGetErrorString(e));
  }
  const int nst = first_step ? 1 : 0;
  CK(cudaMemcpy(sc + r.off_nst, &nst, sizeof(int), cudaMemcpyHostToDevice));
  const size_t zsm = zpass_smem(prec, d->K0, r.z_ppt, r.z_nt);
  const size_t xfs = xpass_smem(prec, (size_t)r.xf_nb * r.X);
  const size_t xis = xpass_smem(prec, (size_t)3 * r.xi_nb * r.X);
  for (int s = 0; s < nsteps; ++s) {
    e = prec == MWF_FP64 ? launch_x_forward_f64(r.x_nt, d_desc, d_items, n_xf, xfs, d_err, st)
                         : launch_x_forward_f32(r.x_nt, d_desc, d_items, n_xf, xfs, d_err, st);
    if (e == cudaSuccess)
      e = prec == MWF_FP64 ? launch_z_nonlinear_f64(d->K0, r.z_ppt, r.z_nt, d_desc, d_items + n_xf, n_z, zsm, d_err, st)
                           : launch_z_nonlinear_f32(d->K0, r.z_ppt, r.z_nt, d_desc, d_items + n_xf, n_z, zsm, d_err, st);
    if (e == cudaSuccess)
      e = prec == MWF_FP64 ? launch_x_inverse_f64(r.x_nt, d_desc, d_items + n_xf + n_z, n_xi, xis, d_err, st)
                           : launch_x_inverse_f32(r.x_nt, d_desc, d_items + n_xf + n_z, n_xi, xis, d_err, st);
    if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_step_noalloc: pass launch: %s", cudaGetErrorString(e));
    CK(cudaMemsetAsync(sc + r.off_nst, 0, sizeof(int), st));
  }
  // a pass that recorded an error skipped work: leave the caller's arrays as they were
  int herr = 0;
  CK(cudaMemcpy(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (herr) return fail(MWF_ERR_DEVICE, "mwf_step_noalloc: kernel reported internal error flags 0x%x", herr);
  // device layout -> caller arrays
  e = prec == MWF_FP64 ? launch_dev_to_ref_f64(sc + r.off_c, c_re, c_im, r.K, r.M, d->NN, st)
                       : launch_dev_to_ref_f32(sc + r.off_c, c_re, c_im, r.K, r.M, d->NN, st);
  if (e == cudaSuccess && nsteps > 0)
    e = prec == MWF_FP64 ? launch_dev_to_ref_f64(sc + r.off_onl, onl_re, onl_im, r.K, r.M, d->NN, st)
                         : launch_dev_to_ref_f32(sc + r.off_onl, onl_re, onl_im, r.K, r.M, d->NN, st);
  if (e != cudaSuccess) return fail(MWF_ERR_CUDA, "mwf_step_noalloc: state conversion: %s", cudaGetErrorString(e));
  CK(cudaStreamSynchronize(st));
  return MWF_OK;
}
