// Backward of the bilinear forms and of the operand folds (FP64, exact).
//
// The forward computes I_L = a^T K_L b (semisep_fp64.cu). K_L is symmetric, so for upstream
// gradients g_L = dLoss/dI_L the operand gradients are
//   dLoss/da = K_g b,   dLoss/db = K_g a,   K_g = sum_L g_L K_L,
// and with the semiseparable structure K_L(p, q) = r_q^L / r_p^(L+1) (q < p), its transpose
// above the diagonal and (1-1e-12)^L / r_p on it:
//   (K_g y)_p = sum_L g_L [ r_p^-(L+1) sum_{q<p} y_q r_q^L + r_p^L sum_{q>p} y_q r_q^-(L+1)
//                           + d_L y_p / r_p ].
// The prefix sums run forward and the suffix sums backward (each is accumulated from its own
// end, so no sum is formed as a difference of totals). K_g b and K_g a are independent: one CTA, half a
// cluster or a cluster of BW_CLUSTER CTAs takes one of them. Every thread owns consecutive points, which
// shared memory holds with their radii and inverse radii (coalesced on the memory side, consecutive on
// the thread side), so the operand is read and the gradient written once.
//
// The folds a = Op (f .* g) (fold.cu) are linear in the product, so dLoss/d(f .* g) = Op^T y
// for y = dLoss/da; the caller multiplies by g and f.
#include <cooperative_groups.h>

#include <utility>

#include "common.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int NL_MAX = 8;       // multipoles per launch (2 scanned series each)
constexpr int BW_THREADS = 128;
constexpr int BW_CLUSTER = 4;   // CTAs per form, or per gradient of a long form
constexpr int BW_CLUSTERS = 148;  // resident clusters: four CTAs of 128 registers and 53 KB per SM
constexpr int BW_NW = BW_THREADS / 32;

// long forms
constexpr int BW_PPT = 16;      // consecutive points per thread
constexpr int BW_WARP = 32 * BW_PPT;          // points per warp and tile
constexpr int BW_TILE = BW_THREADS * BW_PPT;  // points a CTA holds at a time
// shared-memory position of point i of a warp's run: one pad per BW_PPT points, so that the lanes' runs
// of BW_PPT points start in different banks
__device__ __forceinline__ int bw_pos(int i) { return i + i / BW_PPT; }
constexpr int BW_BUF = BW_WARP + BW_WARP / BW_PPT;  // one warp's run of one array
constexpr int BW_HALF_MAX = BW_CLUSTER / 2 * BW_TILE;  // half a cluster holds a form of 4096 points
// short forms: one CTA holds 2048 points, up to 1664 with their inverse radii
constexpr int BW_SEG = 16, BW_SEG_INV = 13;   // points per thread at most
constexpr int BW_SHORT_MAX = BW_SEG * BW_THREADS;
constexpr int BW_SMEM = 4 * BW_SEG_INV * BW_THREADS * (int)sizeof(double);
static_assert(BW_SMEM >= BW_NW * 3 * BW_BUF * (int)sizeof(double), "a tile fits");
static_assert(BW_SMEM >= 3 * (BW_SEG + 1) * BW_THREADS * (int)sizeof(double), "a short form fits");

struct DiagScale {
  double v[DWBA_MAX_L + 1];
};

__device__ __forceinline__ double ipow(double x, int e) {
  double r = 1.0;
  while (e > 0) {
    if (e & 1) r *= x;
    x *= x;
    e >>= 1;
  }
  return r;
}

// What the CTAs of a group share.
template <int NL>
struct Totals {
  static constexpr int NS = 2 * NL;  // scanned series: y r^L (prefix), y r^-(L+1) (suffix)
  double wtot[NS][BW_NW];
  double tot[NS];              // this CTA's totals
  double all[BW_CLUSTER][NS];  // the totals of every CTA of the group, written by it
  double carry[NS];            // series before (prefix) or after (suffix) the tile at hand
};

// One gradient, K_g b (side 0) or K_g a (side 1), by a group of `used` CTAs of a cluster, ranks base .. base + used - 1
// (the other groups of the cluster call it at the same time), each with a consecutive share of the points. FP64
// operations (about 12 per point, multipole and gradient) and the operand traffic (16 bytes per point and gradient)
// bound it about equally. With up to used * BW_TILE points that is one tile and nothing is read twice. Longer forms
// walk their tiles three times (totals, forward with the prefixes, backward with the suffixes).
// 600 forms at N = 6000: 115 us at L <= 4, 149 us at L <= 7 (244 and 292 us with one CTA per form and a strided segment
// per thread). What is left is latency (16 warps per SM: 128 registers, 53 KB), barriers and instruction fetch: a
// second body inline, for forms that do not call it, took 129 and 167 us, so short_gradient is out of line.
template <int NL>
__device__ __forceinline__ void long_gradient(Totals<NL>& S, double* s_buf, const dwba_form_grad_t& F, int side,
                                              int base, int part, int used, const double* __restrict__ grad, int L0,
                                              const DiagScale& ds, int accumulate) {
  constexpr int NW = BW_NW, NS = 2 * NL;
  static_assert(NS * BW_CLUSTER <= BW_THREADS, "one thread per total handed over");
  // another CTA's shared memory may be written once that CTA runs: arrive now, wait before the first write
  cg::cluster_group cluster = cg::this_cluster();
  auto started = cluster.barrier_arrive();
  const double* __restrict__ src = side ? F.a_dev : F.b_dev;
  double* __restrict__ dst = side ? F.gb_dev : F.ga_dev;
  const int n_src = side ? F.n_rows : F.n_cols, n_dst = side ? F.n_cols : F.n_rows;
  const int M = max(n_src, n_dst);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this CTA's points [c0, c1), whole warps' runs so that the loads stay aligned with the lanes
  const int share = ((M + used - 1) / used + BW_WARP - 1) / BW_WARP * BW_WARP;
  const int c0 = min(M, part * share), c1 = min(M, c0 + share);
  const int n_tiles = (c1 - c0 + BW_TILE - 1) / BW_TILE;
  double g[NL];
  double gd = 0.0;  // sum_L g_L d_L over this chunk of multipoles
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    g[l] = grad[l];
    gd += g[l] * ds.v[L0 + l];
  }
  double* sy = s_buf + warp * 3 * BW_BUF;
  double* sr = sy + BW_BUF;
  double* sv = sr + BW_BUF;
  const int own = lane * (BW_PPT + 1);  // bw_pos of the thread's first point
  // the warp's points of tile k into its shared memory; false if the warp has none there
  auto load_tile = [&](int k) -> bool {
    const int w0 = c0 + k * BW_TILE + warp * BW_WARP;
    const int left = c1 - w0;
    if (left <= 0) return false;
    __syncwarp();
    double y[BW_PPT], r[BW_PPT];  // every load is issued before the first is used
#pragma unroll
    for (int j = 0; j < BW_PPT; ++j) {
      const int i = j * 32 + lane;
      y[j] = (i < left && w0 + i < n_src) ? src[w0 + i] : 0.0;
      r[j] = i < left ? F.r_dev[w0 + i] : 1.0;
    }
#pragma unroll
    for (int j = 0; j < BW_PPT; ++j) {
      const int at = bw_pos(j * 32 + lane);
      sy[at] = y[j];
      sr[at] = r[j];
      sv[at] = 1.0 / r[j];
    }
    __syncwarp();
    return true;
  };
  auto pow_lo = [&](double r) { return L0 > 0 ? ipow(r, L0) : 1.0; };  // r^L0
  auto pow_hi = [&](double v) { return L0 > 0 ? ipow(v, L0 + 1) : v; };  // r^-(L0+1), v = 1/r
  // the thread's sums of the prefix series t[0..NL) and of the suffix series t[NL..2NL)
  auto totals = [&](double* t, bool live) {
#pragma unroll
    for (int q = 0; q < NS; ++q) t[q] = 0.0;
    if (!live) return;
#pragma unroll 4
    for (int j = 0; j < BW_PPT; ++j) {
      const double y = sy[own + j], r = sr[own + j], v = sv[own + j];
      double a = y * pow_lo(r), b = y * pow_hi(v);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        t[l] += a;
        t[NL + l] += b;
        a *= r;
        b *= v;
      }
    }
  };
  // exclusive scan of the threads' sums over the tile (prefix series over earlier threads, suffix
  // series over later ones); the warps' totals go to s_wtot (a block-wide call)
  auto scan = [&](double* t, bool live) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const bool up = q < NL;
      double v = t[q];
      if (live) {
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const double u = up ? __shfl_up_sync(0xffffffffu, v, off) : __shfl_down_sync(0xffffffffu, v, off);
          if (up ? lane >= off : lane + off < 32) v += u;
        }
      }
      if (lane == (up ? 31 : 0)) S.wtot[q][warp] = v;
      if (live) {
        const double e = up ? __shfl_up_sync(0xffffffffu, v, 1) : __shfl_down_sync(0xffffffffu, v, 1);
        t[q] = lane == (up ? 0 : 31) ? 0.0 : e;
      }
    }
    __syncthreads();
  };
  // the parts of the warps and tiles before (prefix series) or after (suffix series) this warp
  auto offsets = [&](double* t) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      double o = S.carry[q];
      if (q < NL) {
        for (int w = 0; w < warp; ++w) o += S.wtot[q][w];
      } else {
        for (int w = NW - 1; w > warp; --w) o += S.wtot[q][w];
      }
      t[q] += o;
    }
  };
  auto tile_total = [&](int q) {
    double o = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) o += S.wtot[q][w];
    return o;
  };
  // the carry after the tile at hand (a block-wide call)
  auto advance = [&](int q0, int q1) {
    __syncthreads();
    if (tid >= q0 && tid < q1) S.carry[tid] += tile_total(tid);
    __syncthreads();
  };
  // gradients of the thread's points from the prefix series (forward, with the diagonal) and the
  // suffix series (backward), by Horner's rule over the multipoles
  auto forward = [&](double* t, double* u) {
#pragma unroll
    for (int j = 0; j < BW_PPT; ++j) {
      const double y = sy[own + j], r = sr[own + j], v = sv[own + j];
      double h = 0.0;
#pragma unroll
      for (int l = NL - 1; l >= 0; --l) h = fma(h, v, g[l] * t[l]);
      u[j] = fma(h, pow_hi(v), gd * y * v);
      double a = y * pow_lo(r);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        t[l] += a;
        a *= r;
      }
    }
  };
  auto backward = [&](double* t, double* u) {
#pragma unroll
    for (int j = BW_PPT - 1; j >= 0; --j) {
      const double y = sy[own + j], r = sr[own + j], v = sv[own + j];
      double h = 0.0;
#pragma unroll
      for (int l = NL - 1; l >= 0; --l) h = fma(h, r, g[l] * t[NL + l]);
      u[j] = fma(h, pow_lo(r), u[j]);
      double b = y * pow_hi(v);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        t[NL + l] += b;
        b *= v;
      }
    }
  };
  // the lanes' gradients of tile k to memory
  auto store_tile = [&](int k, const double* u, bool add) {
    const int w0 = c0 + k * BW_TILE + warp * BW_WARP;
#pragma unroll
    for (int j = 0; j < BW_PPT; ++j) sy[own + j] = u[j];  // each lane its own points
    __syncwarp();
#pragma unroll
    for (int j = 0; j < BW_PPT; ++j) {
      const int p = w0 + j * 32 + lane;
      const double x = sy[bw_pos(j * 32 + lane)];
      if (p < c1 && p < n_dst) dst[p] = add ? dst[p] + x : x;
    }
  };

  // 1. the CTA's totals of every series
  double t[NS];
  bool live = false;
  if (tid < NS) S.carry[tid] = 0.0;
  if (n_tiles == 1) {
    live = load_tile(0);
    totals(t, live);
    scan(t, live);  // exclusive within the tile; the other CTAs' parts are added below
    if (tid < NS) S.tot[tid] = tile_total(tid);
  } else {
    for (int k = 0; k < n_tiles; ++k) {
      live = load_tile(k);
      totals(t, live);
      scan(t, live);
      advance(0, NS);
    }
    __syncthreads();
    if (tid < NS) S.tot[tid] = S.carry[tid];
  }
  // 2. every CTA hands its totals to the others (one cluster barrier, no remote loads), then adds the
  // series of the CTAs before (prefix) and after (suffix) it, in order
  __syncthreads();
  cluster.barrier_wait(std::move(started));
  if (tid < NS * used) {
    const int k = tid / NS, q = tid - k * NS;
    *cluster.map_shared_rank(&S.all[part][q], base + k) = S.tot[q];
  }
  cluster.sync();
  if (tid < NS) {
    double o = 0.0;
    if (tid < NL) {
      for (int k = 0; k < part; ++k) o += S.all[k][tid];
    } else {
      for (int k = used - 1; k > part; --k) o += S.all[k][tid];
    }
    S.carry[tid] = o;
  }
  __syncthreads();
  // 3. the gradients
  double u[BW_PPT];
  if (n_tiles == 1) {
    if (live) {
      offsets(t);
      forward(t, u);
      backward(t, u);
      store_tile(0, u, accumulate != 0);
    }
    return;
  }
  for (int k = 0; k < n_tiles; ++k) {
    live = load_tile(k);
    totals(t, live);
    scan(t, live);
    if (live) {
      offsets(t);
      forward(t, u);
      store_tile(k, u, accumulate != 0);
    }
    advance(0, NL);
  }
  for (int k = n_tiles - 1; k >= 0; --k) {
    live = load_tile(k);
    totals(t, live);
    scan(t, live);
    if (live) {
      offsets(t);
#pragma unroll
      for (int j = 0; j < BW_PPT; ++j) u[j] = 0.0;
      backward(t, u);
      store_tile(k, u, true);
    }
    advance(NL, NS);
  }
}

// One gradient of a short form by one CTA: a segment of seg consecutive points per thread (an odd stride apart, so
// that the threads' segments start in different banks), the segments' series scanned by eight threads each. A scan over
// the lanes costs a warp some 500 instructions whatever its points are; this one costs a tenth, and no point is padded.
// Above 1664 points the inverse radii do not fit and are formed again where they are used.
// 600 forms at N = 1500: 31 us at L <= 4, 35 us at L <= 7, 83 us at L <= 10 (47, 51 and 107 us with one CTA for both
// gradients, the segments read from memory).
constexpr int BW_SCAN = BW_THREADS + 8;  // a series' entries, a pad per 16
static_assert(NL_MAX * 8 <= BW_THREADS && NL_MAX * BW_SCAN <= BW_SHORT_MAX, "the series fit");

// exclusive sums over the threads of NL series, in ascending (prefix) or descending order of threads
template <int NL>
__device__ __forceinline__ void thread_scan(double* s, double* v, bool prefix) {
  const int tid = threadIdx.x;
  const int me = prefix ? tid : BW_THREADS - 1 - tid;
  __syncthreads();
#pragma unroll
  for (int l = 0; l < NL; ++l) s[l * BW_SCAN + me + (me >> 4)] = v[l];
  __syncthreads();
  {  // eight threads per series, sixteen entries each
    const int q = tid >> 3, j = tid & 7;
    double* p = s + q * BW_SCAN + 17 * j;
    double sum = 0.0;
    if (q < NL) {
#pragma unroll
      for (int i = 0; i < 16; ++i) sum += p[i];
    }
    double before = sum;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, before, off, 8);
      if (j >= off) before += u;
    }
    before = __shfl_up_sync(0xffffffffu, before, 1, 8);
    if (j == 0) before = 0.0;
    __syncwarp();
    if (q < NL) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const double x = p[i];
        p[i] = before;
        before += x;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int l = 0; l < NL; ++l) v[l] = s[l * BW_SCAN + me + (me >> 4)];
}

template <int NL>
__device__ __noinline__ void short_gradient(double* s_buf, const dwba_form_grad_t* __restrict__ form, int side,
                                            const double* __restrict__ grad, double gd, int L0, int accumulate) {
  const dwba_form_grad_t F = *form;
  const double* __restrict__ src = side ? F.a_dev : F.b_dev;
  double* __restrict__ dst = side ? F.gb_dev : F.ga_dev;
  const int n_src = side ? F.n_rows : F.n_cols, n_dst = side ? F.n_cols : F.n_rows;
  const int M = max(n_src, n_dst), tid = threadIdx.x;
  const int seg = (M + BW_THREADS - 1) / BW_THREADS, stride = seg | 1;
  double* sy = s_buf;
  const bool inv = seg <= BW_SEG_INV;
  const int len = (inv ? BW_SEG_INV : BW_SEG + 1) * BW_THREADS;
  double* sr = sy + len;
  double* su = sr + len;  // the scans, then the gradient
  double* sv = su + len;  // 1/r, if it fits
  const unsigned per = (65536u + seg - 1) / (seg > 0 ? seg : 1);  // i / seg = i * per >> 16 for i < BW_SHORT_MAX
  auto at = [&](int i) { return i + (int)((unsigned)i * per >> 16) * (stride - seg); };
  {
    double y[BW_SEG], r[BW_SEG];  // every load is issued before the first is used
#pragma unroll
    for (int j = 0; j < BW_SEG; ++j) {
      const int i = j * BW_THREADS + tid;
      y[j] = i < n_src ? src[i] : 0.0;
      r[j] = i < M ? F.r_dev[i] : 1.0;
    }
#pragma unroll
    for (int j = 0; j < BW_SEG; ++j) {
      const int i = j * BW_THREADS + tid;
      if (i < M) {
        sy[at(i)] = y[j];
        sr[at(i)] = r[j];
        if (inv) sv[at(i)] = 1.0 / r[j];
      }
    }
  }
  double g[NL], P[NL], S[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    g[l] = grad[l];
    P[l] = S[l] = 0.0;
  }
  const int own = tid * stride, n = max(0, min(seg, M - tid * seg));
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const double y = sy[own + j], r = sr[own + j], v = inv ? sv[own + j] : 1.0 / r;
    double a = y * (L0 > 0 ? ipow(r, L0) : 1.0), b = y * (L0 > 0 ? ipow(v, L0 + 1) : v);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      P[l] += a;
      S[l] += b;
      a *= r;
      b *= v;
    }
  }
  thread_scan<NL>(su, P, true);
  thread_scan<NL>(su, S, false);
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const double y = sy[own + j], r = sr[own + j], v = inv ? sv[own + j] : 1.0 / r;
    double h = 0.0;
#pragma unroll
    for (int l = NL - 1; l >= 0; --l) h = fma(h, v, g[l] * P[l]);
    su[own + j] = fma(h, L0 > 0 ? ipow(v, L0 + 1) : v, gd * y * v);
    double a = y * (L0 > 0 ? ipow(r, L0) : 1.0);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      P[l] += a;
      a *= r;
    }
  }
  for (int j = n - 1; j >= 0; --j) {
    const double y = sy[own + j], r = sr[own + j], v = inv ? sv[own + j] : 1.0 / r;
    double h = 0.0;
#pragma unroll
    for (int l = NL - 1; l >= 0; --l) h = fma(h, r, g[l] * S[l]);
    su[own + j] = fma(h, L0 > 0 ? ipow(r, L0) : 1.0, su[own + j]);
    double b = y * (L0 > 0 ? ipow(v, L0 + 1) : v);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      S[l] += b;
      b *= v;
    }
  }
  __syncthreads();
  for (int i = tid; i < n_dst; i += BW_THREADS) dst[i] = accumulate ? dst[i] + su[at(i)] : su[at(i)];
}

// One launch takes forms of every length without knowing them: two clusters per form, of which a form takes what it
// fills; the other CTAs leave at once (a cluster barrier counts the threads that have not exited). Up to 2048 points a
// CTA has a gradient to itself, above that half a cluster, above 4096 points a cluster. The CTAs that leave are what is
// lost to one CTA per form: below about 800 points and from about 300 forms on that was faster (600 forms at N = 600,
// L <= 7: 21 us, 19 us with one CTA per form; at N = 300: 18 us, 13 us; a second launch for such forms costs every call
// 4 us). Measured against it at 288 sizes, N = 830..6000, 20..600 forms, L <= 2..10, this takes 0.62 of the time in the
// geometric mean and 1.1 of it at most from 1000 points on.
template <int NL>
__global__ void __cluster_dims__(BW_CLUSTER, 1, 1) __launch_bounds__(BW_THREADS, 4)
semisep_backward_kernel(const dwba_form_grad_t* __restrict__ forms, const double* __restrict__ grad, int L0,
                        int n_ltot, DiagScale ds, int accumulate, int few) {
  extern __shared__ double s_buf[];  // per warp: operand, radius, 1/radius of its points
  __shared__ Totals<NL> S;
  const int rank = (int)cg::this_cluster().block_rank();
  const int item = blockIdx.x / BW_CLUSTER, form = item >> 1;
  const dwba_form_grad_t F = forms[form];
  const int M = max(F.n_rows, F.n_cols);
  const int used = M <= BW_SHORT_MAX ? 1 : M <= BW_HALF_MAX ? BW_CLUSTER / 2 : BW_CLUSTER;
  // both gradients in the first of the two clusters where they fit it, unless the GPU has room for one in each (few)
  const bool both = used < BW_CLUSTER && !few;
  if (both ? (item & 1) || rank >= 2 * used : rank >= used) return;
  const int side = both ? rank / used : item & 1, base = both ? rank / used * used : 0;
  const double* g = grad + (int64_t)form * n_ltot + L0;
  if (M <= BW_SHORT_MAX) {
    double gd = 0.0;
#pragma unroll
    for (int l = 0; l < NL; ++l) gd += g[l] * ds.v[L0 + l];
    short_gradient<NL>(s_buf, forms + form, side, g, gd, L0, accumulate);
  } else {
    long_gradient<NL>(S, s_buf, F, side, base, rank - base, used, g, L0, ds, accumulate);
  }
}

template <int NL>
int launch(const dwba_form_grad_t* forms, int n, const double* grad, int L0, int n_ltot, const DiagScale& ds,
           int acc, cudaStream_t st) {
  if (cudaFuncSetAttribute(semisep_backward_kernel<NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, BW_SMEM) !=
      cudaSuccess)
    return DWBA_ERR_CUDA;
  // the grid's x extent is limited to 2^31 - 1 CTAs
  constexpr int MAX_FORMS = 0x7fffffff / (2 * BW_CLUSTER);
  for (int s0 = 0; s0 < n; s0 += MAX_FORMS) {
    const int m = n - s0 < MAX_FORMS ? n - s0 : MAX_FORMS;
    semisep_backward_kernel<NL><<<m * 2 * BW_CLUSTER, BW_THREADS, BW_SMEM, st>>>(
        forms + s0, grad + (int64_t)s0 * n_ltot, L0, n_ltot, ds, acc, 2 * m <= BW_CLUSTERS);
    DWBA_CHECK_LAUNCH();
  }
  return DWBA_OK;
}

int launch_nl(int nl, const dwba_form_grad_t* forms, int n, const double* grad, int L0, int n_ltot,
              const DiagScale& ds, int acc, cudaStream_t st) {
  switch (nl) {
#define DWBA_CASE(N) \
  case N: return launch<N>(forms, n, grad, L0, n_ltot, ds, acc, st);
    DWBA_CASE(1) DWBA_CASE(2) DWBA_CASE(3) DWBA_CASE(4) DWBA_CASE(5) DWBA_CASE(6) DWBA_CASE(7) DWBA_CASE(8)
#undef DWBA_CASE
    default: return DWBA_ERR_INVALID_ARG;
  }
}

// z = Op^T y for one fold; Op row i holds the taps of columns i-H..i+H
__global__ void fold_adjoint_kernel(const dwba_fold_adj_t* __restrict__ adj) {
  const dwba_fold_adj_t A = adj[blockIdx.y];
  const int H = A.half_band, W = 2 * H + 1;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < A.n_src; k += gridDim.x * blockDim.x) {
    double z = 0.0;
    for (int d = -H; d <= H; ++d) {
      const int i = k - d;  // row whose tap d reaches column k
      if (i >= 0 && i < A.n_out) z += A.op_dev[(int64_t)W * i + (d + H)] * A.y_dev[i];
    }
    A.z_dev[k] = z;
  }
}

}  // namespace

extern "C" int dwba_bilinear_semisep_backward_fp64(const dwba_form_grad_t* forms_dev, int n_forms, int L_max,
                                                   const double* diag_scale_host, const double* grad_dev,
                                                   double r_min_all, double r_max_all, dwba_stream_t stream) {
  if (n_forms <= 0) return DWBA_OK;
  if (!forms_dev || !diag_scale_host || !grad_dev || L_max < 0 || L_max > DWBA_MAX_L || !(r_min_all > 0.0) ||
      !(r_max_all >= r_min_all) || n_forms > 0x7fffffff)
    return DWBA_ERR_INVALID_ARG;
  const double lmin = log10(r_min_all), lmax = log10(r_max_all);
  const double worst = fmax(fabs(lmin) * (L_max + 1), fabs(lmax) * (L_max + 1));
  if (worst > 280.0) return DWBA_ERR_UNSUPPORTED;
  DiagScale ds;
  for (int l = 0; l <= DWBA_MAX_L; ++l) ds.v[l] = l <= L_max ? diag_scale_host[l] : 0.0;
  const int n_ltot = L_max + 1;
  const int chunks = (n_ltot + NL_MAX - 1) / NL_MAX;  // of about equal size: the largest have the most spills
  for (int c = 0, L0 = 0; c < chunks; ++c) {
    const int nl = (n_ltot - L0 + chunks - c - 1) / (chunks - c);
    const int rc = launch_nl(nl, forms_dev, n_forms, grad_dev, L0, n_ltot, ds, L0 > 0 ? 1 : 0,
                             (cudaStream_t)stream);
    if (rc != DWBA_OK) return rc;
    L0 += nl;
  }
  return DWBA_OK;
}

extern "C" int dwba_fold_adjoint(const dwba_fold_adj_t* adj_dev, int n, int max_len, dwba_stream_t stream) {
  if (n <= 0) return DWBA_OK;
  if (!adj_dev || max_len < 0 || n > 65535) return DWBA_ERR_INVALID_ARG;
  dim3 grid(dwba_grid_1d(max_len, 256, 1024), n);
  fold_adjoint_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(adj_dev);
  DWBA_CHECK_LAUNCH();
  return DWBA_OK;
}
