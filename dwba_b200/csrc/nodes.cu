// Node-set operators: the phase-split Clenshaw-Curtis quadrature of the
// reference folded into banded matrices on the radial grid.
//
// Reference semantics (oscillatory_integrals.py):
//   * breakpoints: generate_phase_nodes (:1625-1713) -- linspace for eta == 0
//     (rebuilt here on the device with numpy's linspace arithmetic), host list otherwise;
//   * CC nodes of interval [a, b]: x = hw*(x_ref+1) + a, W = w_ref*hw, hw = 0.5*(b-a),
//     intervals with b - a <= 1e-12 skipped (:2578-2601, :2701-2712);
//   * outer interpolation P1: _interp_on_radial_grid on r[:n1] (:279-302);
//   * exchange: rho2 interpolated by P2 on the full grid, kernel columns by
//     linear-in-r weights Q with idx_right = clip(searchsorted(r, x), 1, N-1) (:2714-2742).
// With these, the reference's outer sum sum_c W_c (P1 rho1)_c (P1 v)_c equals
// rho1^T T v, T = P1^T diag(W) P1 (tridiagonal), and the exchange inner sum
// sum_c K(r_i, x_c) W_c (P2 rho2)_c equals sum_k K_ik (B rho2)_k with
// B = Q^T diag(W) P2 (band of half-width 2).
//
// Every CC node lies in one grid interval (r_g, r_{g+1}] and feeds only rows g and
// g+1, so one thread per grid interval evaluates the nodes it owns once
// (enumerating the phase intervals that overlap its grid interval and recomputing
// their nodes with the reference's arithmetic), sums their contributions per
// target row, and each row adds the sums of its two owners through warp shuffles
// (deterministic, no scratch memory, no atomics). Where phase intervals of equal
// width lie wholly inside a grid interval (72-82 % of the nodes of the measured
// batch), their sums are formed in closed form.
#include "phase_nodes.cuh"

namespace {

using namespace dwba_nodes;

// 1/x for 1e-30 < x < 1e30 by two Newton-Raphson steps from the single-precision reciprocal: within an ulp,
// and a third of the instructions of a division
__device__ __forceinline__ double recip(double x) {
  const float f = (float)x;
  if (!(f > 1e-30f && f < 1e30f)) return 1.0 / x;
  double y = (double)(1.0f / f);
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// log(1 + u) for 0 <= u <= 1/64 by its Taylor series in Estrin form (shorter dependency chains
// than Horner): 6 terms for u <= 2^-9, 12 terms up to 1/64 (truncation below 1e-17 relative).
__device__ __forceinline__ double log1p_series6(double u) {
  const double u2 = u * u;
  const double e0 = fma(-0.5, u, 1.0), e1 = fma(-0.25, u, 1.0 / 3.0), e2 = fma(-1.0 / 6.0, u, 0.2);
  return u * fma(fma(e2, u2, e1), u2, e0);
}
__device__ __forceinline__ double log1p_series12(double u) {
  const double u2 = u * u, u4 = u2 * u2;
  const double e0 = fma(-0.5, u, 1.0), e1 = fma(-0.25, u, 1.0 / 3.0), e2 = fma(-1.0 / 6.0, u, 0.2);
  const double e3 = fma(-0.125, u, 1.0 / 7.0), e4 = fma(-0.1, u, 1.0 / 9.0), e5 = fma(-1.0 / 12.0, u, 1.0 / 11.0);
  const double lo = fma(fma(e2, u2, e1), u2, e0);
  const double hi = fma(fma(e5, u2, e4), u2, e3);
  return u * fma(hi, u4 * u2, lo);
}

// Sums over a run of M whole phase intervals of equal width 2 hw inside one interpolation interval
// [r_g, r_{g+1}], in closed form. With s = (x - r_g)/(r_{g+1} - r_g), a node is s = s_c + e, s_c the centre
// of the run, e = eta (2j - (M-1) + x_q) for interval j and reference node x_q (eta = hw / (r_{g+1} - r_g)).
// The Clenshaw-Curtis rule is symmetric, so the odd powers of e cancel and the even ones are
//   D_i = sum w e^i = hw eta^i sum_j sum_q w_q (2j - (M-1) + x_q)^i,
// polynomials in M with the rule's moments W_i = sum_q w_q x_q^i. The log tap is, exactly to rounding,
//   t = t0 + tau(e),  tau = T1 (e - v e^2/2 + v^2 e^3/3 - ...),  T1 = v / (log r_{g+1} - log r_g),
//   v = (r_{g+1} - r_g) / (r_g + s_c (r_{g+1} - r_g)) <= 1/64, |e| <= 1/2: the terms past e^8 are below 1e-18
// (past e^6 for steps up to 2^-9); a linear tap has v = 0, T1 = 1. All sums a row needs follow from
//   A = sum w tau,  Bq = sum w tau^2,  C = sum w e tau.
// Weight and centre of the run are those of its ends as rounded, to which the rounded intervals add up; inside
// it the positions are the exact ones, where a node by itself rounds to an ulp of x.
struct RunTaps {
  double t0, A, Bq, C;
};

__device__ __forceinline__ RunTaps run_taps(const double* __restrict__ W, double M, double hw, double eta, double t0,
                                            double T1, double v, bool short6) {
  RunTaps R;
  const double m2 = M * M, e = eta * eta, y = e * v * v;
  const double S2 = M * (m2 - 1.0) * (1.0 / 3.0);
  const double S4 = S2 * fma(3.0, m2, -7.0) * 0.2;
  const double S6 = S2 * fma(fma(3.0, m2, -18.0), m2, 31.0) * (1.0 / 7.0);
  const double he = hw * e;
  const double D2 = he * fma(S2, W[0], M * W[1]);
  const double G4 = he * y * fma(S4, W[0], fma(6.0 * S2, W[1], M * W[2]));
  const double G6 = he * y * y * fma(S6, W[0], fma(15.0 * S4, W[1], fma(15.0 * S2, W[2], M * W[3])));
  // by powers of e: sum w tau / (T1 v), sum w tau^2 / T1^2, sum w e tau / T1
  double a = fma(-1.0 / 6.0, G6, fma(-0.25, G4, -0.5 * D2));
  double b = fma(0.4 + 0.25 + 1.0 / 9.0, G6, fma(2.0 / 3.0 + 0.25, G4, D2));
  double c = fma(0.2, G6, fma(1.0 / 3.0, G4, D2));
  if (!short6) {
    const double S8 = S2 * fma(fma(fma(5.0, m2, -55.0), m2, 239.0), m2, -381.0) * (1.0 / 15.0);
    const double G8 = he * y * y * y *
                      fma(S8, W[0], fma(28.0 * S6, W[1], fma(70.0 * S4, W[2], fma(28.0 * S2, W[3], M * W[4]))));
    a = fma(-0.125, G8, a);
    b = fma(2.0 / 7.0 + 1.0 / 6.0 + 2.0 / 15.0 + 0.0625, G8, b);
    c = fma(1.0 / 7.0, G8, c);
  }
  R.t0 = t0;
  R.A = T1 * v * a;
  R.Bq = T1 * T1 * b;
  R.C = T1 * c;
  return R;
}

// One warp per CTA covers OWN_ROWS consecutive grid rows. Lane j owns grid interval
// g = k0 - 1 + j: the CC nodes whose kernel-column interval (searchsorted left, clipped) is
// il = g, i.e. x in (r_g, r_{g+1}] (g = 0: [r_0, r_1]). Each node is evaluated once, by its
// owner, and reaches rows g and g+1; the owner sums them per target row, and row k adds the sums of
// lanes k-1 and k through warp shuffles. Lane 0 is the halo of the first row (its own row is written by
// the previous CTA).
//
// With t the (log-)interpolation weight in interval g, wr the linear column weight and w the CC weight, a
// node adds
//   T: row g += w(1-t)^2 (diagonal), w(1-t)t (upper); row g+1 += wt^2 (diagonal), wt(1-t) (lower)
//   B: row g += (1-wr) w(1-t2), (1-wr) w t2 (taps 0, 1); row g+1 += wr w(1-t2), wr w t2 (taps -1, 0).
// A node exactly at r_{g+1} is interpolated in interval g+1 with t = 0 (or, at the end of the range, in
// interval g with t = 1): the same entries either way, w on row g+1's diagonal of T and its column weights
// on tap 1 of row g and tap 0 of row g+1. So T is symmetric (one sum serves both off-diagonals) and B has
// taps -1, 0 and 1.
constexpr int OWN_ROWS = 31;
// A CTA (one warp) takes one set and strides over its row blocks: consecutive row blocks of a set run at the
// same time, and the costly ones (many nodes per grid interval) are spread over the CTAs. (Walking over the
// sets with a fixed row block, which keeps the grid's reciprocals and the bound functions' rows: 1.77 ms
// against 1.50 ms on the 2048-set batch.) Latency bounds it: 32 resident warps per SM at 64 registers
// are worth their spills (1.50 ms; 1.60 at 72 registers, 1.79 at 80 without most of the spills, 1.98 at 96).
// The batch (2048 sets, N = 15000, four transitions): 2.36 ms node by node with a factor's fold loads at a
// time, 1.93 ms with whole intervals in closed form, 1.50 ms with two off-diagonals and a tap fewer and
// Newton-Raphson reciprocals, 1.37 ms with the fold's loads together and prefetched.
#ifndef DWBA_NODESET_FILL
#define DWBA_NODESET_FILL 32 // resident-CTA waves the launch aims for
#endif
#ifndef DWBA_NODESET_PREFETCH
#define DWBA_NODESET_PREFETCH 1
#endif
#ifndef DWBA_NODESET_FC
#define DWBA_NODESET_FC 5  // factors whose loads are in flight together (1: 1.46 ms, 2: 1.38, 3: 1.38, 5: 1.37)
#endif
#ifndef DWBA_NODESET_MIN_BLOCKS
#define DWBA_NODESET_MIN_BLOCKS 24
#endif
#ifndef DWBA_NODESET_FOLD_MIN_BLOCKS
#define DWBA_NODESET_FOLD_MIN_BLOCKS 32
#endif
// FOLD = true: the operators are not stored; each row applies them at once to the two multi-folds
// of its set (folds[2 set] with the tridiagonal T, folds[2 set + 1] with the band B, taps -1, 0 and 1),
// with the arithmetic of fold_multi_kernel, and writes the folded operands instead.
__device__ __forceinline__ void fold_row_from_taps(const dwba_fold_multi_t& m, int i, double* tap) {
  if (i >= m.n_clear) return;
  const int n_f = m.n_f, n_src = m.n_src;
  if (i >= m.n_out) {
    for (int t = 0; t < n_f; ++t) m.out_dev[t][i] = 0.0;
    return;
  }
  const double* __restrict__ g = m.g_dev + i;
  if (i >= 1 && i + 1 < n_src) {  // inside: no bounds per tap
#pragma unroll
    for (int d = 0; d < 3; ++d) tap[d] *= g[d - 1];
    // the loads of FC factors in flight; streaming stores: the folded operands are read by the next kernels
    // from DRAM
    constexpr int FC = DWBA_NODESET_FC;
#pragma unroll 1
    for (int t0 = 0; t0 < n_f; t0 += FC) {
      double fv[FC][3];
#pragma unroll
      for (int c = 0; c < FC; ++c) {
        const double* __restrict__ f = m.f_dev[min(t0 + c, n_f - 1)] + i;
#pragma unroll
        for (int d = 0; d < 3; ++d) fv[c][d] = f[d - 1];
      }
#pragma unroll
      for (int c = 0; c < FC; ++c)
        if (t0 + c < n_f)
          __stcs(m.out_dev[t0 + c] + i, fma(tap[2], fv[c][2], fma(tap[1], fv[c][1], tap[0] * fv[c][0])));
    }
    return;
  }
  for (int t = 0; t < n_f; ++t) {
    const double* __restrict__ f = m.f_dev[t] + i;
    double acc = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int k = i + d - 1;
      if (k >= 0 && k < n_src) acc = fma(tap[d] * g[d - 1], f[d - 1], acc);
    }
    __stcs(m.out_dev[t] + i, acc);
  }
}

// Bring the rows k0 - 1 .. k0 + 31 of the functions a row block's folds read into L1 while its nodes are
// summed: at the fold, one factor's loads at a time would each wait for L2 or DRAM.
__device__ __forceinline__ void prefetch_rows(const dwba_fold_multi_t* fm, int k0, int lane) {
  const int lines = 3;  // 128-byte lines of 33 rows
  const int nT = fm[0].n_f + 1, total = (nT + fm[1].n_f + 1) * lines;
  for (int i = lane; i < total; i += 32) {
    const int a = i / lines, line = i - a * lines;
    const dwba_fold_multi_t& m = fm[a < nT ? 0 : 1];
    const int q = a < nT ? a : a - nT;  // 0: g, else factor q - 1
    const double* p = q == 0 ? m.g_dev : m.f_dev[q - 1];
    const int row = min(max(k0 - 1, 0) + line * 16, m.n_src - 1);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p + row));
  }
}

template <int NCC, bool FOLD>  // NCC: CC nodes per interval known at compile time (0: n_cc at run time)
__global__ void __launch_bounds__(32, FOLD ? DWBA_NODESET_FOLD_MIN_BLOCKS : DWBA_NODESET_MIN_BLOCKS)
    nodeset_rows_kernel(const dwba_nodeset_t* __restrict__ sets, const double* __restrict__ ccx_g,
                        const double* __restrict__ ccw_g, int n_cc_rt, const dwba_fold_multi_t* __restrict__ folds) {
  __shared__ double ccw[MAX_CC], ccx1[MAX_CC];
  __shared__ double cc_mom[5];  // sum_q w_q x_q^(2 i)
  // the set's two multi-fold descriptors (T, then B), read by every row of the CTA
  __shared__ dwba_fold_multi_t fm[FOLD ? 2 : 1];
  const int n_cc = NCC > 0 ? NCC : n_cc_rt;
  const int lane = threadIdx.x;
  if (lane < n_cc) {
    ccw[lane] = ccw_g[lane];
    ccx1[lane] = rn_add(ccx_g[lane], 1.0);
  }
  const double ccx_q = lane < n_cc ? ccx_g[lane] : 0.0, ccw_q = lane < n_cc ? ccw_g[lane] : 0.0;
  const double ccx_m = lane < n_cc ? ccx_g[n_cc - 1 - lane] : 0.0, ccw_m = lane < n_cc ? ccw_g[n_cc - 1 - lane] : 0.0;
  const bool cc_sym = __all_sync(0xffffffffu, fabs(ccx_q + ccx_m) <= 1e-15 && fabs(ccw_q - ccw_m) <= 1e-15 * fabs(ccw_q));
  {
    double p = ccw_q;
    for (int i = 0; i < 5; ++i) {
      double v = p;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) cc_mom[i] = v;
      p *= ccx_q * ccx_q;
    }
  }
  if (FOLD) {
    constexpr int W = (int)(2 * sizeof(dwba_fold_multi_t) / sizeof(unsigned long long));
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(folds + 2 * (int64_t)blockIdx.y);
    for (int w = lane; w < W; w += 32) reinterpret_cast<unsigned long long*>(fm)[w] = src[w];
  }
  __syncwarp();
  const dwba_nodeset_t d = sets[blockIdx.y];
  const int N = d.n_grid, n1 = d.n1;
  const double* __restrict__ r = d.r_dev;
  SetView s;
  s.r = r;
  s.br = d.breaks_dev;
  s.n_int = d.n_breaks - 1;
  s.log1 = d.log1;
  s.log2 = d.log2;
  s.start = r[0];
  s.stop = r[n1 - 1];
  s.step = rn_sub(s.stop, s.start) / (double)s.n_int;
  s.inv_step = recip(s.step);
  const bool any_log = s.log1 || s.log2;
  // runs of whole intervals in closed form: equal intervals (linspace), a symmetric rule
  const bool runs = s.br == nullptr && cc_sym && s.step > 1e-11;

  for (int k0 = blockIdx.x * OWN_ROWS; k0 < N; k0 += gridDim.x * OWN_ROWS) {
    const int g = k0 - 1 + lane;
    const double rg = r[min(max(g, 0), N - 1)];
    if (FOLD && DWBA_NODESET_PREFETCH) prefetch_rows(fm, k0, lane);
    // sums for row g (o_*) and row g+1 (x_*); o_up is also row g+1's lower off-diagonal of T
    double o_di = 0.0, o_up = 0.0, x_di = 0.0, o_b2 = 0.0, o_b3 = 0.0, x_b1 = 0.0, x_b2 = 0.0;
    const int m_first = interval_floor(s, rg);
    // the last interval that starts at or below r_{g+1}: the next lane's first
    int m_last = __shfl_down_sync(0xffffffffu, m_first, 1);
    // nodes lie in [r_0, r_{n1-1}], so owners stop at g = n1 - 2
    if (g >= 0 && g <= n1 - 2) {
      const double rg1 = r[g + 1];
      if (lane == 31 && runs) m_last = interval_floor(s, rg1);
      const double lo = g == 0 ? -1.0e308 : rg;  // exclusive lower end of the owned interval
      const double dr = rg1 - rg;
      const double irg = recip(rg), iW = recip(dr + 1e-30);
      const double il = any_log ? recip(d.logr_dev[g + 1] - d.logr_dev[g]) : 0.0;
      const double iT = s.log1 ? il : iW, iB = s.log2 ? il : iW;
      const double u_max = dr * irg;
      const bool short6 = u_max <= 0.001953125;
      const bool series = u_max <= 0.015625;  // every log tap of the interval by its series
      double b = interval_start(s, m_first);
      for (int m = m_first; m < s.n_int; ++m) {
        const double a = b;  // one interval's end is the next one's start
        if (a > rg1) break;
        b = interval_end(s, m);
        if (runs && m == m_first + 1 && m < m_last && (!any_log || series)) {
          // whole intervals strictly inside: m .. m_end (the last one ends below r_{g+1})
          int m_end = m_last - 1;
          double be = interval_end(s, m_end);
          if (be >= rg1) be = interval_end(s, --m_end);
          if (m_end >= m) {
            const double hw = 0.5 * s.step, M = (double)(m_end - m + 1);
            // the intervals' widths and centres add up to the run's ends as they are rounded
            const double D0 = 0.5 * (be - a) * cc_mom[0];
            const double xc = 0.5 * ((a - rg) + (be - rg));
            const double sc = xc * iW, uc = xc * irg, eta = hw * iW;
            const double l1 = any_log ? (short6 ? log1p_series6(uc) : log1p_series12(uc)) : 0.0;
            const double v = any_log ? u_max * recip(1.0 + uc) : 0.0;
            RunTaps R = s.log1 ? run_taps(cc_mom, M, hw, eta, l1 * iT, v * iT, v, short6)
                               : run_taps(cc_mom, M, hw, eta, sc, 1.0, 0.0, true);
            double c = 1.0 - R.t0;
            o_di += fma(c * c, D0, fma(-2.0 * c, R.A, R.Bq));
            o_up += fma(c - R.t0, R.A, fma(R.t0 * c, D0, -R.Bq));
            x_di += fma(R.t0 * R.t0, D0, fma(2.0 * R.t0, R.A, R.Bq));
            if (s.log2 != s.log1) {
              R = s.log2 ? run_taps(cc_mom, M, hw, eta, l1 * iB, v * iB, v, short6)
                         : run_taps(cc_mom, M, hw, eta, sc, 1.0, 0.0, true);
              c = 1.0 - R.t0;
            }
            const double d = 1.0 - sc, wo = fma(c, D0, -R.A), wt = fma(R.t0, D0, R.A);
            o_b2 += fma(d, wo, R.C);
            o_b3 += fma(d, wt, -R.C);
            x_b1 += fma(sc, wo, -R.C);
            x_b2 += fma(sc, wt, R.C);
            m = m_end;
            b = be;
            continue;
          }
        }
        const double width = rn_sub(b, a);
        if (!(width > 1e-12)) continue;
        const double hw = rn_mul(0.5, width);
        // kept rolled: unrolled it spills at this register budget
#pragma unroll 1
        for (int q = 0; q < (NCC > 0 ? NCC : MAX_CC); ++q) {  // ascending positions within the interval
          if (NCC == 0 && q >= n_cc) break;
          const int sl = n_cc - 1 - q;
          double x = rn_add(rn_mul(hw, ccx1[sl]), a);  // >= a
          if (sl == 0) x = fmin(x, b);  // the top node can round one ulp past b
          if (!(x > lo)) continue;
          if (x > rg1) break;  // as are all later ones
          const double w = rn_mul(ccw[sl], hw);
          const double dx = x - rg;
          const double q1 = dx * iW, q0 = 1.0 - q1;
          if (x >= rg1) {  // exactly at r_{g+1}
            x_di += w;
            o_b3 = fma(q0, w, o_b3);
            x_b2 = fma(q1, w, x_b2);
            continue;
          }
          // log x - log r_g: from the series of log(1 + (x - r_g)/r_g) when the grid step is small (it
          // then equals the difference of the two logs to a few ulps of that difference), else as the
          // difference
          double dl = 0.0;
          if (any_log) {
            const double u = dx * irg;
            dl = short6 ? log1p_series6(u) : (u <= 0.015625 ? log1p_series12(u) : log(x) - d.logr_dev[g]);
          }
          const double t = s.log1 ? dl * iT : dx * iT;
          const double omt = 1.0 - t;
          double wo = w * omt, wt = w * t;
          o_di = fma(wo, omt, o_di);
          o_up = fma(wo, t, o_up);
          x_di = fma(wt, t, x_di);
          if (s.log1 != s.log2) {
            const double t2 = s.log2 ? dl * iB : dx * iB;
            wo = w * (1.0 - t2);
            wt = w * t2;
          }
          o_b2 = fma(q0, wo, o_b2);
          o_b3 = fma(q0, wt, o_b3);
          x_b1 = fma(q1, wo, x_b1);
          x_b2 = fma(q1, wt, x_b2);
        }
      }
    }
    // row g = sums of lane - 1 (its row g+1) and of this lane, in that order
    const double t0 = __shfl_up_sync(0xffffffffu, o_up, 1);  // from nodes below r_g only
    const double t1 = __shfl_up_sync(0xffffffffu, x_di, 1) + o_di;
    const double b1 = __shfl_up_sync(0xffffffffu, x_b1, 1);
    const double b2 = __shfl_up_sync(0xffffffffu, x_b2, 1) + o_b2;
    if (lane >= 1 && g < N) {
      if (FOLD) {
        if (g < n1) {
          double tt[3] = {t0, t1, o_up};
          fold_row_from_taps(fm[0], g, tt);
        }
        double bb[3] = {b1, b2, o_b3};
        fold_row_from_taps(fm[FOLD ? 1 : 0], g, bb);
      } else {
        if (g < n1) {
          d.ta_dev[3 * g + 0] = t0;
          d.ta_dev[3 * g + 1] = t1;
          d.ta_dev[3 * g + 2] = o_up;
        }
        double* bx = d.bx_dev + 5 * (int64_t)g;
        bx[0] = 0.0;
        bx[1] = b1;
        bx[2] = b2;
        bx[3] = o_b3;
        bx[4] = 0.0;
      }
    }
  }
}

// row groups per set: enough warps in total to fill the GPU several times over, never more than
// the largest set needs (each warp strides over its set's row blocks)
dim3 nodeset_grid(int max_grid, int n_sets) {
  const int need = (max_grid + OWN_ROWS - 1) / OWN_ROWS;
  const int fill = (int)(((int64_t)148 * 24 * DWBA_NODESET_FILL + n_sets - 1) / n_sets);
  return dim3(need < fill ? need : fill, n_sets);
}

}  // namespace

extern "C" int dwba_build_nodesets(const dwba_nodeset_t* sets_dev, int n_sets, int max_grid, const double* cc_x_dev,
                                   const double* cc_w_dev, int n_cc, int* /*status_dev*/, dwba_stream_t stream) {
  if (n_sets <= 0) return DWBA_OK;
  if (!sets_dev || !cc_x_dev || !cc_w_dev || n_cc < 2 || n_cc > MAX_CC || max_grid < 2 ||
      n_sets > 65535)
    return DWBA_ERR_INVALID_ARG;
  const dim3 grid = nodeset_grid(max_grid, n_sets);
  if (n_cc == 5)
    nodeset_rows_kernel<5, false><<<grid, 32, 0, (cudaStream_t)stream>>>(sets_dev, cc_x_dev, cc_w_dev, n_cc, nullptr);
  else
    nodeset_rows_kernel<0, false><<<grid, 32, 0, (cudaStream_t)stream>>>(sets_dev, cc_x_dev, cc_w_dev, n_cc, nullptr);
  DWBA_CHECK_LAUNCH();
  return DWBA_OK;
}

extern "C" int dwba_build_nodesets_folded(const dwba_nodeset_t* sets_dev, const dwba_fold_multi_t* folds_dev,
                                          int n_sets, int max_grid, const double* cc_x_dev, const double* cc_w_dev,
                                          int n_cc, int* /*status_dev*/, dwba_stream_t stream) {
  if (n_sets <= 0) return DWBA_OK;
  if (!sets_dev || !folds_dev || !cc_x_dev || !cc_w_dev || n_cc < 2 || n_cc > MAX_CC ||
      max_grid < 2 || n_sets > 65535)
    return DWBA_ERR_INVALID_ARG;
  const dim3 grid = nodeset_grid(max_grid, n_sets);
  if (n_cc == 5)
    nodeset_rows_kernel<5, true><<<grid, 32, 0, (cudaStream_t)stream>>>(sets_dev, cc_x_dev, cc_w_dev, n_cc, folds_dev);
  else
    nodeset_rows_kernel<0, true><<<grid, 32, 0, (cudaStream_t)stream>>>(sets_dev, cc_x_dev, cc_w_dev, n_cc, folds_dev);
  DWBA_CHECK_LAUNCH();
  return DWBA_OK;
}
