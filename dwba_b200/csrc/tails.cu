// Outer tails of the direct integral on the GPU: one CTA per (pair, chunk of up to 8 multipoles). The Filon
// panels of a phase branch are equal, so their sum is one sum over its nodes: the alpha terms of neighbouring
// panels cancel, an inner node between panels has weight 2 beta, one inside a panel gamma, and the
// envelope powers are advanced node by node with one multiply-add per multipole (the moments enter once at
// the end). The threads take runs of nodes; each Levin segment's factorised collocation system serves every
// multipole of the chunk.
//
// Same quantity and formulas as the host path (host.cpp, dwba_outer_tails), which follows
// oscillatory_integrals.py: dwba_outer_integral_1d (:459-535) with
// compute_outer_integral_oscillatory (:1361-1451: Filon when |Phi''| h^2 < 0.1, else Levin),
// _filon_segment_complex (:1165-1277), _levin_segment_complex (:1024-1095) and
// _analytical_multipole_tail (:2064-2184). The reference sums segment contributions with
// math.fsum; here a thread's runs (16 nodes at most, plain sums) and its Levin and low-frequency segments enter a
// compensated sum, the threads' sums are added by warp shuffles and the warps' in order.
// Pairs whose mid-interval frequency is below 1e-10 (the reference's adaptive-quadrature
// branch) are left to the host path: the caller routes them there.
#include "common.cuh"

namespace {

struct cplx {
  double re, im;
};
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx cscale(double s, cplx a) { return {s * a.re, s * a.im}; }
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  const double d = b.re * b.re + b.im * b.im;
  return {(a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d};
}
__device__ __forceinline__ cplx cexpi(double phi) {
  double s, c;
  sincos(phi, &s, &c);
  return {c, s};
}

struct WaveD {
  double k, delta, eta, sigma;
  int l;
};

struct PhaseD {
  WaveD a, b;
  int sgn;
  double kk, cc;
  __device__ PhaseD(const WaveD& wa, const WaveD& wb, int s) : a(wa), b(wb), sgn(s) {
    const double ca = -a.l * M_PI / 2 + a.sigma + a.delta;
    const double cb = -b.l * M_PI / 2 + b.sigma + b.delta;
    kk = s < 0 ? a.k - b.k : a.k + b.k;
    cc = s < 0 ? ca - cb : ca + cb;
  }
  __device__ double phi(double r) const {
    double v = kk * r + cc;
    if (fabs(a.eta) > 1e-15) v += a.eta * log(2 * a.k * r + 1e-30);
    if (fabs(b.eta) > 1e-15) {
      const double t = b.eta * log(2 * b.k * r + 1e-30);
      v = sgn < 0 ? v - t : v + t;
    }
    if (a.l > 0) v -= (a.l * (a.l + 1)) / (2.0 * a.k * r);
    if (b.l > 0) {
      const double t = (b.l * (b.l + 1)) / (2.0 * b.k * r);
      v = sgn < 0 ? v + t : v - t;
    }
    return v;
  }
  __device__ double d1(double r) const {
    double v = kk;
    if (fabs(a.eta) > 1e-15) v += a.eta / r;
    if (fabs(b.eta) > 1e-15) v = sgn < 0 ? v - b.eta / r : v + b.eta / r;
    if (a.l > 0) v += (a.l * (a.l + 1)) / (2.0 * a.k * (r * r));
    if (b.l > 0) {
      const double t = (b.l * (b.l + 1)) / (2.0 * b.k * (r * r));
      v = sgn < 0 ? v - t : v + t;
    }
    return v;
  }
  __device__ double d2(double r) const {
    double v = 0.0;
    if (fabs(a.eta) > 1e-15) v -= a.eta / (r * r);
    if (fabs(b.eta) > 1e-15) v = sgn < 0 ? v + b.eta / (r * r) : v - b.eta / (r * r);
    const double r3 = r * r * r;
    if (a.l > 0) v -= (a.l * (a.l + 1)) / (a.k * r3);
    if (b.l > 0) {
      const double t = (b.l * (b.l + 1)) / (b.k * r3);
      v = sgn < 0 ? v + t : v - t;
    }
    return v;
  }
};

// numpy.linspace(a, b, n)[i]
__device__ __forceinline__ double lin(double a, double b, int n, int i) {
  if (i == n - 1) return b;
  return (double)i * ((b - a) / (double)(n - 1)) + a;
}

// 1/x for 1e-30 < x < 1e30 by two Newton-Raphson steps from the single-precision reciprocal (within an ulp)
__device__ __forceinline__ double tail_recip(double x) {
  const float f = (float)x;
  if (!(f > 1e-30f && f < 1e30f)) return 1.0 / x;
  double y = (double)(1.0f / f);
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// compensated lane sum
struct KSum {
  double s = 0.0, c = 0.0;
  __device__ void add(double x) {
    const double t = s + x;
    if (fabs(s) >= fabs(x)) c += (s - t) + x; else c += (x - t) + s;
    s = t;
  }
};

struct LevinD {
  double D[8][8];  // Chebyshev differentiation matrix of descending Lobatto points (reference convention)
  double xr[8];    // ascending reference nodes in [-1, 1]
};

__shared__ LevinD s_lv;  // the launch's Levin tables, staged once per block

__device__ double warp_sum(double v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

constexpr int LC = 8;  // multipoles evaluated together (one accumulator each per lane)
constexpr int TAIL_THREADS = 128;

// b^e for e >= 0 by repeated squaring
__device__ __forceinline__ double ipow(double b, int e) {
  double r = 1.0;
  while (e) {
    if (e & 1) r *= b;
    b *= b;
    e >>= 1;
  }
  return r;
}

// x^-(L0+1) for the envelopes f_L(x) = m_L x^-(L+1) of a chunk (0 where x <= 1e-6): the envelope of
// multipole L0 + q is m[q] p with p advanced by 1/x per multipole
struct EnvPow {
  double p0, inv;
  __device__ __forceinline__ EnvPow(double x, int L0) {
    const bool in = x > 1e-6;
    inv = in ? 1.0 / x : 0.0;
    p0 = in ? ipow(inv, L0 + 1) : 0.0;
  }
};

// Filon constants shared by every panel of one phase branch: the segments are equal (linspace) and
// so are their panels, so alpha, beta, gamma of the panel angle theta = omega h / 2 and the phase
// step between nodes, E = exp(i omega h / 2), are evaluated once per branch instead of per panel.
struct FilonConst {
  double al, be, ga;
  cplx E;
};

__device__ __forceinline__ FilonConst filon_const(double omega, double seg_w, int nn) {
  FilonConst c;
  const double h = 2.0 * seg_w / (nn - 1);  // panel width (two node spacings)
  const double th = omega * h / 2;
  double st, ct;
  sincos(th, &st, &ct);
  c.E = {ct, st};
  if (fabs(th) < 0.3) {
    const double t2 = th * th, t3 = t2 * th, t6 = t2 * t2 * t2;
    c.al = 2 * t3 / 45 * (1 - t2 / 7 + (t2 * t2) / 189);
    c.be = 2.0 / 3 + 2 * t2 / 15 - 4 * (t2 * t2) / 105 + 2 * t6 / 567;
    c.ga = 4.0 / 3 - 2 * t2 / 15 + 1 * (t2 * t2) / 210 - t6 / 11340;
  } else {
    const double t2 = th * th, t3 = t2 * th;
    double s2, c2;
    sincos(2 * th, &s2, &c2);
    c.al = (t2 + th * s2 / 2 - 2 * (st * st)) / t3;
    c.be = 2 * (th * (1 + c2) - s2) / t3;
    c.ga = 4 * (st - th * ct) / t3;
  }
  return c;
}

// Re of the Filon integral over one segment (nn equally spaced nodes, nn odd) for every multipole
// of the chunk: _filon_segment_complex with the node phases and the panel weights shared by all L.
// The first node's phase factor is evaluated directly, the next ones by the recurrence
// e_{j+1} = e_j E (nn - 1 <= 14 steps: a few ulps), and the panels use the branch's FilonConst.
// Envelope values are formed inside the multipole loops from one running power per node, so no
// per-node arrays of envelopes are kept.
__device__ __forceinline__ void filon_segment_all(const double* m, int L0, int nl, double a, double b, int nn, double omega,
                                  double off, const FilonConst& fc, KSum* acc) {
  if (!(b - a >= 1e-15)) return;
  if (fabs(omega * (b - a)) < 1e-3) {  // scipy simpson with possibly unequal spacing, times the mid phase
    const double ce = cexpi(omega * (a + b) / 2 + off).re;
    double part[LC];
#pragma unroll
    for (int q = 0; q < LC; ++q) part[q] = 0.0;
    for (int i = 0; i + 2 < nn; i += 2) {
      const double x0 = lin(a, b, nn, i), x1 = lin(a, b, nn, i + 1), x2 = lin(a, b, nn, i + 2);
      const double h0 = x1 - x0, h1 = x2 - x1;
      const double hs = h0 + h1, hp = h0 * h1, qq = h0 / h1;
      const EnvPow e0(x0, L0), e1(x1, L0), e2(x2, L0);
      double p0 = e0.p0, p1 = e1.p0, p2 = e2.p0;
#pragma unroll
      for (int q = 0; q < LC; ++q) {
        const double mq = q < nl ? m[q] : 0.0;
        part[q] += hs / 6.0 * ((mq * p0) * (2.0 - 1.0 / qq) + (mq * p1) * (hs * (hs / hp)) + (mq * p2) * (2.0 - qq));
        p0 *= e0.inv;
        p1 *= e1.inv;
        p2 *= e2.inv;
      }
    }
#pragma unroll
    for (int q = 0; q < LC; ++q) acc[q].add(part[q] * ce);
    return;
  }
  double seg[LC];
#pragma unroll
  for (int q = 0; q < LC; ++q) seg[q] = 0.0;
  double x0 = a;
  cplx e0 = cexpi(omega * x0 + off);
  EnvPow v0(x0, L0);
  const cplx mi = {0.0, -1.0 / omega};
  const cplx am = cscale(fc.al, mi);
  const cplx wl = csub(cplx{fc.be, 0.0}, am), wr = cadd(cplx{fc.be, 0.0}, am);
  for (int i = 0; i + 2 < nn; i += 2) {
    const double x1 = lin(a, b, nn, i + 1), x2 = lin(a, b, nn, i + 2);
    const double h = x2 - x0;
    const cplx e1 = cmul(e0, fc.E), e2 = cmul(e1, fc.E);
    const EnvPow v1(x1, L0), v2(x2, L0);
    if (h >= 1e-15) {
      double w0, w1, w2;
      if (fabs(omega * h) < 1e-3) {  // the 3-node panel itself is non-oscillatory: Simpson times the mid phase
        const double h0 = x1 - x0, h1 = x2 - x1;
        const double hs = h0 + h1, hp = h0 * h1, qq = h0 / h1;
        const double ce = cexpi(omega * (x0 + x2) / 2 + off).re;
        w0 = ce * (hs / 6.0) * (2.0 - 1.0 / qq);
        w1 = ce * (hs / 6.0) * (hs * (hs / hp));
        w2 = ce * (hs / 6.0) * (2.0 - qq);
      } else {
        // (h/2) [alpha (-i/omega) (f2 e2 - f0 e0) + beta (f0 e0 + f2 e2) + gamma f1 e1], real part,
        // as weights of f0, f1, f2 that every multipole shares
        w0 = (h / 2) * cmul(wl, e0).re;
        w1 = (h / 2) * (fc.ga * e1.re);
        w2 = (h / 2) * cmul(wr, e2).re;
      }
      double p0 = v0.p0, p1 = v1.p0, p2 = v2.p0;
#pragma unroll
      for (int q = 0; q < LC; ++q) {
        const double mq = q < nl ? m[q] : 0.0;
        seg[q] += w0 * (mq * p0) + w1 * (mq * p1) + w2 * (mq * p2);
        p0 *= v0.inv;
        p1 *= v1.inv;
        p2 *= v2.inv;
      }
    }
    x0 = x2;
    e0 = e2;
    v0 = v2;
  }
#pragma unroll
  for (int q = 0; q < LC; ++q) acc[q].add(seg[q]);
}

// sum of w_j cos(omega x_j + off) x_j^-(L+1) over the nodes j0 .. j1-1 of a branch's n_int equal intervals of
// width d (n_int even), w_j the composite Filon weights without the factor h/2: a direct phase for the first
// node, then the recurrence e_{j+1} = e_j E (runs of at most FILON_RUN nodes: a few ulps).
constexpr int FILON_RUN = 16;
template <int NL>
__device__ __forceinline__ void filon_run(int L0, double rm, double d, int n_int, int j0, int j1, double omega,
                                          double off, const FilonConst& fc, double* sum) {
  // the run's first phase omega (rm + j0 d) + off with the roundings of its three operations put back: they
  // are some 1e-14 at a phase of hundreds, and the whole run would share them
  const double p0 = (double)j0 * d, pe = fma((double)j0, d, -p0);
  double x = rm + p0;
  const double bv = x - rm, xe = ((rm - (x - bv)) + (p0 - bv)) + pe;
  const double w0 = omega * x, we = fma(omega, x, -w0) + omega * xe;
  const double f0 = w0 + off, bf = f0 - w0, fe = ((w0 - (f0 - bf)) + (off - bf)) + we;
  cplx e = cexpi(f0);
  e = {fma(-fe, e.im, e.re), fma(fe, e.re, e.im)};
#pragma unroll
  for (int q = 0; q < NL; ++q) sum[q] = 0.0;
#pragma unroll 2
  for (int j = j0; j < j1; ++j) {
    double w = (j & 1) ? fc.ga * e.re : 2.0 * fc.be * e.re;
    if (j == 0) w = fc.be * e.re - fc.al / omega * e.im;
    if (j == n_int) w = fc.be * e.re + fc.al / omega * e.im;
    double p = 0.0, inv = 0.0;
    if (x > 1e-6) {  // (the envelope is cut there)
      inv = tail_recip(x);
      p = inv * inv;
      for (int k = 1; k < L0; ++k) p *= inv;
    }
#pragma unroll
    for (int q = 0; q < NL; ++q) {
      sum[q] = fma(w, p, sum[q]);
      p *= inv;
    }
    e = {fma(e.re, fc.E.re, -e.im * fc.E.im), fma(e.re, fc.E.im, e.im * fc.E.re)};
    x = fma((double)(j + 1), d, rm);
  }
}

// Levin collocation on one segment (8 nodes) for every multipole of the chunk, solved by a group
// of 8 lanes: lane `row` of the group holds row `row` of the 8x8 complex collocation system in
// registers (compile-time column indices only, so nothing goes to local memory). The system does
// not depend on L: it is factorised once by Gaussian elimination with partial pivoting (largest
// |re| + |im| of the column among the rows not yet used; the pivot order is kept instead of
// swapping rows, and the pivot row is broadcast by shuffles) and solved for each envelope.
// All 32 lanes call it together (shuffles over groups of 8); `valid` = the group has a segment.
// res[q]: the segment's contribution to multipole L0 + q, the same on every lane of the group
// (zero for an invalid group or a singular system).
__device__ __noinline__ void levin_segment_group(const double* m, int L0, int nl, const PhaseD& ph, double a, double b,
                                                 bool valid, double* res) {
  const int row = threadIdx.x & 7;
  const LevinD& lv = s_lv;
  const double hw = 0.5 * (b - a);
  const double xi = hw * (lv.xr[row] + 1) + a;
  const double x0 = hw * (lv.xr[0] + 1) + a, x7 = hw * (lv.xr[7] + 1) + a;
  const double h = x7 - x0;
  bool ok = valid && !(h < 1e-15);
  const double sc = ok ? 2.0 / h : 0.0;
  const double d1 = ph.d1(xi);
  cplx A[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) A[j] = {lv.D[row][j] * sc, j == row ? d1 : 0.0};
  int step_of = 8;  // elimination step at which this row became the pivot
  int pv[8];        // pivot row of each step
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double mag = step_of < 8 ? -1.0 : fabs(A[k].re) + fabs(A[k].im);
    int who = row;
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {  // group argmax, ties to the lower row
      const double om = __shfl_xor_sync(0xffffffffu, mag, off, 8);
      const int ow = __shfl_xor_sync(0xffffffffu, who, off, 8);
      if (om > mag || (om == mag && ow < who)) {
        mag = om;
        who = ow;
      }
    }
    pv[k] = who;
    if (!(mag > 0.0)) ok = false;  // singular (or an invalid group): the result is dropped
    cplx P[8];
#pragma unroll
    for (int j = k; j < 8; ++j) {
      P[j].re = __shfl_sync(0xffffffffu, A[j].re, who, 8);
      P[j].im = __shfl_sync(0xffffffffu, A[j].im, who, 8);
    }
    if (row == who) {
      step_of = k;
    } else if (step_of == 8) {
      const cplx inv = cdiv({1.0, 0.0}, P[k]);
      const cplx l = cmul(A[k], inv);
      A[k] = l;
#pragma unroll
      for (int j = k + 1; j < 8; ++j) A[j] = csub(A[j], cmul(l, P[j]));
    }
  }
  const cplx e7 = cexpi(ph.phi(x7)), e0 = cexpi(ph.phi(x0));
  const double inv_x = xi > 1e-6 ? 1.0 / xi : 0.0;
  double pw = xi > 1e-6 ? ipow(inv_x, L0 + 1) : 0.0;
#pragma unroll 1
  for (int q = 0; q < LC; ++q) {
    res[q] = 0.0;
    if (q >= nl) continue;  // warp-uniform
    cplx u = {m[q] * pw, 0.0};
    pw *= inv_x;
    // forward: rows that became pivots after step k take their multiplier of step k
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      cplx y;
      y.re = __shfl_sync(0xffffffffu, u.re, pv[k], 8);
      y.im = __shfl_sync(0xffffffffu, u.im, pv[k], 8);
      if (step_of > k) u = csub(u, cmul(A[k], y));
    }
    // backward: the pivot row of step k gives unknown k (node k); every lane keeps all unknowns
    cplx z[8];
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      cplx t = u;
#pragma unroll
      for (int j = k + 1; j < 8; ++j) t = csub(t, cmul(A[j], z[j]));
      const cplx zk = cdiv(t, A[k]);
      z[k].re = __shfl_sync(0xffffffffu, zk.re, pv[k], 8);
      z[k].im = __shfl_sync(0xffffffffu, zk.im, pv[k], 8);
    }
    res[q] = ok ? csub(cmul(z[7], e7), cmul(z[0], e0)).re : 0.0;
  }
}

// What a phase branch's threads share: its constant frequency and offset, the segments and the Filon constants
struct BranchPlan {
  double om, off, eff;
  FilonConst fc;
  int filon, nseg, nn;
};

__device__ __noinline__ BranchPlan plan_branch(const PhaseD& ph, double rm, double rmax, int max_seg, double max_dphi) {
  BranchPlan B;
  const double delta_phi = M_PI / 4;
  B.om = fabs(ph.d1((rm + rmax) / 2));
  const double h = delta_phi / B.om;
  B.filon = fabs(ph.d2((rm + rmax) / 2)) * h * h < 0.1 ? 1 : 0;
  B.off = B.eff = 0.0;
  B.nn = 5;
  B.fc = FilonConst{0.0, 0.0, 0.0, {1.0, 0.0}};
  if (B.filon) {
    B.off = ph.phi(rm) - B.om * rm;
    const double dr = delta_phi / B.om;
    const long long nraw = max(1LL, (long long)ceil((rmax - rm) / dr));
    B.nseg = (int)min(nraw, (long long)max_seg);
    B.eff = B.om * (rmax - rm) / max(1, B.nseg);
    if (B.eff > max_dphi) {
      const int scl = (int)ceil(B.eff / max_dphi);
      B.nn = min(15, max(5, 5 + 2 * (scl - 1)));
    }
    B.fc = filon_const(B.om, (rmax - rm) / B.nseg, B.nn);
  } else {
    B.nseg = (int)max(1.0, ceil((rmax - rm) / h));
  }
  return B;
}

__device__ __forceinline__ WaveD wave_of(const dwba_tail_t* R, int w) {
  const double* v = R->wave + 5 * w;
  return {v[0], v[2], v[3], v[4], (int)v[1]};
}

// The Levin segments of a branch, or the segments of a branch whose panels hardly oscillate, times
// sgn, into sum (a CTA-wide call): rare, and kept out of the Filon path's registers
__device__ __noinline__ void other_segments(const double* m, int L0, int nl, const PhaseD& ph, const BranchPlan& B,
                                            double rm, double rmax, double sgn, double* sum) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nseg = B.nseg;
  KSum acc[LC];
  if (B.filon) {
    for (int s = tid; s < nseg; s += TAIL_THREADS) {
      const double a = lin(rm, rmax, nseg + 1, s), b = lin(rm, rmax, nseg + 1, s + 1);
      filon_segment_all(m, L0, nl, a, b, B.nn, B.om, B.off, B.fc, acc);
    }
  } else {
    // four segments per warp pass, one per group of 8 lanes; lane 0 of a group accumulates it
    const int grp = lane >> 3;
    for (int s0 = 4 * warp; s0 < nseg; s0 += TAIL_THREADS / 8) {  // warp-uniform
      const int s = s0 + grp;
      const bool valid = s < nseg;
      const double a = valid ? lin(rm, rmax, nseg + 1, s) : rm;
      const double b = valid ? lin(rm, rmax, nseg + 1, s + 1) : rm;
      double res[LC];
      levin_segment_group(m, L0, nl, ph, a, b, valid, res);
      if (valid && (lane & 7) == 0) {
#pragma unroll
        for (int q = 0; q < LC; ++q)
          if (q < nl) acc[q].add(res[q]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < LC; ++q) sum[q] = sgn * (acc[q].s + acc[q].c);
}

// one phase branch (cos(Phi_a -/+ Phi_b)) of the outer integral for a chunk of multipoles, times sgn, added to
// the threads' sums (a CTA-wide call)
template <int NL>
__device__ __forceinline__ void branch_sum(const double* m, int L0, int nl, const dwba_tail_t* R, int sign,
                                           const BranchPlan& B, double rm, double rmax, double sgn, KSum* acc) {
  if (B.filon && B.eff >= 0.01) {  // every panel oscillates (its phase is eff 2/(nn-1) >= 1e-3)
    const int tid = threadIdx.x;
    const FilonConst fc = B.fc;
    const int n_int = B.nseg * (B.nn - 1);
    const double d = (rmax - rm) / n_int;
    const int rounds = (n_int + 1 + TAIL_THREADS * FILON_RUN - 1) / (TAIL_THREADS * FILON_RUN);
    const int len = (n_int + 1 + TAIL_THREADS * rounds - 1) / (TAIL_THREADS * rounds);
    for (int k = 0; k < rounds; ++k) {
      const int j0 = (k * TAIL_THREADS + tid) * len, j1 = min(j0 + len, n_int + 1);
      if (j0 >= j1) break;
      double sum[NL];
      filon_run<NL>(L0, rm, d, n_int, j0, j1, B.om, B.off, fc, sum);
#pragma unroll
      for (int q = 0; q < NL; ++q) acc[q].add(sgn * d * m[q] * sum[q]);  // h/2 = d
    }
    return;
  }
  double mm[LC], sum[LC];
#pragma unroll
  for (int q = 0; q < LC; ++q) mm[q] = q < NL ? m[q] : 0.0;
  const PhaseD ph(wave_of(R, 0), wave_of(R, 1), sign);
  other_segments(mm, L0, nl, ph, B, rm, rmax, sgn, sum);
#pragma unroll
  for (int q = 0; q < NL; ++q) acc[q].add(sum[q]);
}

__device__ double analytical_tail(double r_m, const WaveD& wi, const WaveD& wf, int L, double overlap) {
  if (r_m < 1e-3 || fabs(overlap) < 1e-12) return 0.0;
  const double lti = fabs(wi.eta) > 1e-10 ? wi.eta * log(2 * wi.k * r_m + 1e-30) : 0.0;
  const double ltf = fabs(wf.eta) > 1e-10 ? wf.eta * log(2 * wf.k * r_m + 1e-30) : 0.0;
  const double ci = -wi.l * M_PI / 2 + wi.sigma + wi.delta + lti;
  const double cf = -wf.l * M_PI / 2 + wf.sigma + wf.delta + ltf;
  const double kd = wi.k - wf.k, ks = wi.k + wf.k;
  const int n = L + 1;
  const double rn = ipow(r_m, n);  // r_m^n
  double t = 0.0;
  const double pd = kd * r_m + ci - cf;
  if (fabs(kd) > 1e-6) {
    t += 0.5 * (sin(pd) / (kd * rn) + n * cos(pd) / ((kd * kd) * (rn * r_m)));
  } else if (n > 1) {
    t += 0.5 * cos(pd) / ((n - 1) * ipow(r_m, n - 1));
  }
  const double ps = ks * r_m + ci + cf;
  if (ks > 1e-6) t -= 0.5 * (sin(ps) / (ks * rn) + n * cos(ps) / ((ks * ks) * (rn * r_m)));
  if (!isfinite(t)) return 0.0;
  return t * overlap;
}

// A CTA takes `per` consecutive items (a record and a chunk of up to NL multipoles): first the constants of all
// their phase branches, one branch per thread (a dozen transcendental functions each); then item by item both
// branches over all threads, one after the other (they differ widely in length), with one reduction; last the
// analytical tails, one (item, multipole) per thread. NL: the chunk's multipoles, or LC.
// Bound by the dependent chains of the runs and the issue of their FP64 operations: 13,407 records, L <= 6, in
// 330 us (775 us with a warp per record, segment by segment with three weights a panel; 569 us with every thread
// forming the branches' constants), 150 records in 22 us (105 us).
constexpr int TAIL_ITEMS = TAIL_THREADS / 2;  // at most
constexpr int TAIL_FILL = 20;  // CTAs per SM the launch aims for (8: 378 us, 16: 331, 24: 329, 32: 352)

template <int NL>
__global__ void __launch_bounds__(TAIL_THREADS, 4)
tails_kernel(const dwba_tail_t* __restrict__ recs, int n, int L_max, int max_seg, double max_dphi, int per, LevinD lv) {
  __shared__ double s_red[TAIL_THREADS / 32][NL];
  __shared__ double s_t[TAIL_ITEMS][NL];
  __shared__ BranchPlan s_plan[TAIL_THREADS];
  for (int i = threadIdx.x; i < 72; i += blockDim.x)
    (&s_lv.D[0][0])[i] = i < 64 ? lv.D[i / 8][i % 8] : lv.xr[i - 64];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_chunk = (L_max + LC - 1) / LC;
  const int64_t n_items = (int64_t)n * n_chunk;
  for (int64_t it0 = (int64_t)blockIdx.x * per; it0 < n_items; it0 += (int64_t)gridDim.x * per) {
    const int cnt = (int)min((int64_t)per, n_items - it0);
    __syncthreads();  // the previous items' plans and sums are consumed
    if (tid < 2 * cnt) {
      const dwba_tail_t* R = recs + (it0 + tid / 2) / n_chunk;
      if (R->mode != 1)
        s_plan[tid] = plan_branch(PhaseD(wave_of(R, 0), wave_of(R, 1), (tid & 1) ? +1 : -1), R->r_m, R->r_max, max_seg,
                                  max_dphi);
    }
    __syncthreads();
    for (int k = 0; k < cnt; ++k) {
      const int rec = (int)((it0 + k) / n_chunk);
      const int L0 = 1 + (int)(it0 + k - (int64_t)rec * n_chunk) * LC;  // multipoles L0 .. L0+nl-1
      const int nl = min(NL, L_max + 1 - L0);
      const dwba_tail_t* R = recs + rec;
      const double r_m = R->r_m, r_max = R->r_max;
      double m[NL];
      bool any = false;
#pragma unroll
      for (int q = 0; q < NL; ++q) {
        const double v = q < nl ? R->moments_dev[L0 + q] : 0.0;
        m[q] = fabs(v) > 1e-12 ? v : 0.0;  // moments at or below the cut-off give a zero tail
        any = any || m[q] != 0.0;
      }
      KSum acc[NL];
      if (any && R->mode != 1 && !(r_max <= r_m + 1e-10)) {  // uniform over the CTA
#pragma unroll 1
        for (int br = 0; br < 2; ++br)
          branch_sum<NL>(m, L0, nl, R, br ? +1 : -1, s_plan[2 * k + br], r_m, r_max, br ? -0.5 : 0.5, acc);
      }
#pragma unroll
      for (int q = 0; q < NL; ++q) {
        const double v = warp_sum(acc[q].s + acc[q].c);
        if (lane == 0) s_red[warp][q] = v;
      }
      __syncthreads();
      if (tid < NL) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < TAIL_THREADS / 32; ++w) t += s_red[w][tid];
        s_t[k][tid] = t;
      }
      __syncthreads();
    }
    for (int i = tid; i < cnt * NL; i += TAIL_THREADS) {
      const int k = i / NL, q = i - k * NL;
      const int rec = (int)((it0 + k) / n_chunk);
      const int L = 1 + (int)(it0 + k - (int64_t)rec * n_chunk) * LC + q;
      if (L > L_max) continue;
      const dwba_tail_t* R = recs + rec;
      const double v = R->moments_dev[L];
      double o = 0.0;
      if (fabs(v) > 1e-12) {
        const WaveD wi = wave_of(R, 0), wf = wave_of(R, 1);
        o = R->mode == 1 ? analytical_tail(R->r_m, wi, wf, L, v) : s_t[k][q] + analytical_tail(R->r_max, wi, wf, L, v);
      }
      R->out_dev[L] = o;
      if (L == 1) R->out_dev[0] = 0.0;
    }
  }
}

template <int NL>
void launch_tails(const dwba_tail_t* recs, int n, int L_max, int max_seg, double max_dphi, const LevinD& lv,
                  cudaStream_t st) {
  // one item per CTA until they fill the GPU, then up to TAIL_ITEMS (what an item's threads sum does not
  // depend on it)
  const int64_t items = (int64_t)n * ((L_max + LC - 1) / LC);
  const int64_t want = items / (148 * TAIL_FILL);
  const int per = (int)(want < 1 ? 1 : (want > TAIL_ITEMS ? TAIL_ITEMS : want));
  tails_kernel<NL><<<dwba_grid_1d(items, per, 1 << 30), TAIL_THREADS, 0, st>>>(recs, n, L_max, max_seg, max_dphi, per, lv);
}

}  // namespace

extern "C" int dwba_outer_tails_batch(const dwba_tail_t* tails_dev, int n, int L_max, int max_filon_segments,
                                      double max_effective_dphi, dwba_stream_t stream) {
  if (n <= 0 || L_max < 1) return DWBA_OK;
  if (!tails_dev || L_max > DWBA_MAX_L || max_filon_segments < 1 || !(max_effective_dphi > 0.0))
    return DWBA_ERR_INVALID_ARG;
  // Chebyshev differentiation matrix (descending Lobatto points) and ascending nodes, n = 8
  LevinD lv;
  double x[8], c[8];
  for (int i = 0; i < 8; ++i) {
    x[i] = cos(M_PI * i / 7);
    c[i] = (i == 0 || i == 7) ? 2.0 : 1.0;
  }
  for (int i = 0; i < 8; ++i) {
    double rs = 0.0;
    for (int j = 0; j < 8; ++j) {
      if (i == j) continue;
      const double sgn = ((i + j) % 2 == 0) ? 1.0 : -1.0;
      lv.D[i][j] = (c[i] / c[j]) * sgn / (x[i] - x[j]);
      rs += lv.D[i][j];
    }
    lv.D[i][i] = -rs;
  }
  for (int k = 0; k < 8; ++k) lv.xr[k] = cos(M_PI * (7 - k) / 7);
  cudaStream_t st = (cudaStream_t)stream;
  switch (L_max < LC ? L_max : LC) {
#define DWBA_CASE(N) \
  case N: launch_tails<N>(tails_dev, n, L_max, max_filon_segments, max_effective_dphi, lv, st); break;
    DWBA_CASE(1) DWBA_CASE(2) DWBA_CASE(3) DWBA_CASE(4) DWBA_CASE(5) DWBA_CASE(6) DWBA_CASE(7) DWBA_CASE(8)
#undef DWBA_CASE
  }
  DWBA_CHECK_LAUNCH();
  return DWBA_OK;
}
