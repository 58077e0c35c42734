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
// end, so no sum is formed as a difference of totals). K_g b and K_g a are independent: a cluster of
// BW_CLUSTER CTAs takes one of them. Every thread owns BW_PPT consecutive points, which its warp holds
// in shared memory with their radii and inverse radii (coalesced on the memory side, consecutive on
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
constexpr int BW_PPT = 16;      // consecutive points per thread
constexpr int BW_WARP = 32 * BW_PPT;          // points per warp and tile
constexpr int BW_TILE = BW_THREADS * BW_PPT;  // points a CTA holds at a time
constexpr int BW_CLUSTER = 4;   // CTAs per operand gradient
constexpr int BW_NW = BW_THREADS / 32;
// shared-memory position of point i of a warp's run: one pad per BW_PPT points, so that the lanes' runs
// of BW_PPT points start in different banks
__device__ __forceinline__ int bw_pos(int i) { return i + i / BW_PPT; }
constexpr int BW_BUF = BW_WARP + BW_WARP / BW_PPT;  // one warp's run of one array
constexpr int BW_SHORT = 1536, BW_SHORT_FORMS = 200;
constexpr int BW_SMEM = BW_NW * 3 * BW_BUF * (int)sizeof(double);

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

// FP64 operations (about 12 per point, multipole and gradient) and the operand traffic (16 bytes per
// point and gradient) bound it about equally. A CTA owns a consecutive share of the points; with up to
// BW_CLUSTER * BW_TILE = 8192 points that is one tile and nothing is read twice. Longer forms walk
// their tiles three times (totals, forward with the prefixes, backward with the suffixes).
// 676 forms at N = 6000, L <= 4: 122 us (290 us with one CTA per form and a strided segment per thread); 600 forms at
// N = 1500, L <= 6: 72 us (104 us when all four CTAs of a cluster took a share of a short form, a warp of each).
// What is left is latency: 13 warps per SM (128 registers, 52 KB), barriers and instruction fetch.
template <int NL>
__global__ void __cluster_dims__(BW_CLUSTER, 1, 1) __launch_bounds__(BW_THREADS, 4)
semisep_backward_kernel(const dwba_form_grad_t* __restrict__ forms, const double* __restrict__ grad, int L0,
                        int n_ltot, DiagScale ds, int accumulate, int shortest) {
  constexpr int NW = BW_NW;
  constexpr int NS = 2 * NL;  // scanned series: y r^L (prefix), y r^-(L+1) (suffix)
  extern __shared__ double s_buf[];  // per warp: operand, radius, 1/radius of its points
  __shared__ double s_wtot[NS][NW];
  __shared__ double s_tot[NS];    // this CTA's totals
  __shared__ double s_all[BW_CLUSTER][NS];  // every CTA's totals, written by it
  static_assert(NS * BW_CLUSTER <= BW_THREADS, "one thread per total handed over");
  __shared__ double s_carry[NS];  // series before (prefix) or after (suffix) the tile at hand
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int item = blockIdx.x / BW_CLUSTER;
  const int form = item >> 1, side = item & 1;  // side 0: ga = K_g b, side 1: gb = K_g a
  const dwba_form_grad_t F = forms[form];
  const double* __restrict__ src = side ? F.a_dev : F.b_dev;
  double* __restrict__ dst = side ? F.gb_dev : F.ga_dev;
  const int n_src = side ? F.n_rows : F.n_cols, n_dst = side ? F.n_cols : F.n_rows;
  const int M = max(n_src, n_dst);
  // a form takes as many CTAs as it fills with one tile each; the others leave at once (a cluster barrier counts
  // the threads that have not exited)
  const int used = min(BW_CLUSTER, max(1, (M + BW_TILE - 1) / BW_TILE));
  if (rank >= used || M < shortest) return;
  // another CTA's shared memory may be written once that CTA runs: arrive now, wait before the first write
  auto started = cluster.barrier_arrive();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this CTA's points [c0, c1), whole warps' runs so that the loads stay aligned with the lanes
  const int share = ((M + used - 1) / used + BW_WARP - 1) / BW_WARP * BW_WARP;
  const int c0 = min(M, rank * share), c1 = min(M, c0 + share);
  const int n_tiles = (c1 - c0 + BW_TILE - 1) / BW_TILE;
  double g[NL];
  double gd = 0.0;  // sum_L g_L d_L over this chunk of multipoles
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    g[l] = grad[(int64_t)form * n_ltot + L0 + l];
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
      if (lane == (up ? 31 : 0)) s_wtot[q][warp] = v;
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
      double o = s_carry[q];
      if (q < NL) {
        for (int w = 0; w < warp; ++w) o += s_wtot[q][w];
      } else {
        for (int w = NW - 1; w > warp; --w) o += s_wtot[q][w];
      }
      t[q] += o;
    }
  };
  auto tile_total = [&](int q) {
    double o = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) o += s_wtot[q][w];
    return o;
  };
  // the carry after the tile at hand (a block-wide call)
  auto advance = [&](int q0, int q1) {
    __syncthreads();
    if (tid >= q0 && tid < q1) s_carry[tid] += tile_total(tid);
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
  if (tid < NS) s_carry[tid] = 0.0;
  if (n_tiles == 1) {
    live = load_tile(0);
    totals(t, live);
    scan(t, live);  // exclusive within the tile; the other CTAs' parts are added below
    if (tid < NS) s_tot[tid] = tile_total(tid);
  } else {
    for (int k = 0; k < n_tiles; ++k) {
      live = load_tile(k);
      totals(t, live);
      scan(t, live);
      advance(0, NS);
    }
    __syncthreads();
    if (tid < NS) s_tot[tid] = s_carry[tid];
  }
  // 2. every CTA hands its totals to the others (one cluster barrier, no remote loads), then adds the
  // series of the CTAs before (prefix) and after (suffix) it, in order
  __syncthreads();
  cluster.barrier_wait(std::move(started));
  if (tid < NS * used) {
    const int k = tid / NS, q = tid - k * NS;
    *cluster.map_shared_rank(&s_all[rank][q], k) = s_tot[q];
  }
  cluster.sync();
  if (tid < NS) {
    double o = 0.0;
    if (tid < NL) {
      for (int k = 0; k < rank; ++k) o += s_all[k][tid];
    } else {
      for (int k = used - 1; k > rank; --k) o += s_all[k][tid];
    }
    s_carry[tid] = o;
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

// Forms of up to BW_SHORT points when there are BW_SHORT_FORMS of them or more: one CTA per form takes both gradients,
// a strided segment per thread. Such forms fill the chip by their number, and the cluster kernel's CTAs would have few
// points each: 600 forms at N = 1500, L <= 6: 48 us (72 us with the cluster kernel); at N = 2000 it is 104 us against
// 74 us. Fewer forms leave the chip idle either way (100 forms at N = 1500, L <= 10: 43 us and 45 us). The launch
// does not know the forms' lengths, so both kernels are launched and each takes its own.
template <int NL>
__global__ void __launch_bounds__(BW_THREADS)
semisep_backward_short_kernel(const dwba_form_grad_t* __restrict__ forms, const double* __restrict__ grad, int L0,
                        int n_ltot, DiagScale ds, int accumulate) {
  __shared__ double scan[4 * NL][BW_THREADS + 1];
  const dwba_form_grad_t F = forms[blockIdx.x];
  const int M = F.n_rows > F.n_cols ? F.n_rows : F.n_cols;
  if (M > BW_SHORT) return;
  const int tid = threadIdx.x;
  const int seg = (M + BW_THREADS - 1) / BW_THREADS;
  const int p0 = tid * seg;
  const int p1 = min(M, p0 + seg);
  double g[NL];
  double gd = 0.0;  // sum_L g_L d_L over this chunk of multipoles
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    g[l] = grad[(int64_t)blockIdx.x * n_ltot + L0 + l];
    gd += g[l] * ds.v[L0 + l];
  }

  // pass 1: segment totals of a r^L, b r^L (prefix series) and a r^-(L+1), b r^-(L+1) (suffix series)
  double ta[NL], tb[NL], sa[NL], sb[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) ta[l] = tb[l] = sa[l] = sb[l] = 0.0;
  for (int p = p0; p < p1; ++p) {
    const double X = p < F.n_rows ? F.a_dev[p] : 0.0;
    const double Y = p < F.n_cols ? F.b_dev[p] : 0.0;
    const double r = F.r_dev[p], inv = 1.0 / r;
    double pw = L0 > 0 ? ipow(r, L0) : 1.0;
    double ip = L0 > 0 ? ipow(inv, L0 + 1) : inv;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      ta[l] += X * pw;
      tb[l] += Y * pw;
      sa[l] += X * ip;
      sb[l] += Y * ip;
      pw *= r;
      ip *= inv;
    }
  }
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    scan[l][tid] = ta[l];
    scan[NL + l][tid] = tb[l];
    scan[2 * NL + l][tid + 1] = sa[l];
    scan[3 * NL + l][tid + 1] = sb[l];
  }
  __syncthreads();
  if (tid < 2 * NL) {  // exclusive prefix over segments: entry k = sum of segments < k
    double s = 0.0;
    for (int k = 0; k < BW_THREADS; ++k) {
      const double v = scan[tid][k];
      scan[tid][k] = s;
      s += v;
    }
  } else if (tid < 4 * NL) {  // exclusive suffix over segments: entry k+1 = sum of segments > k
    double s = 0.0;
    for (int k = BW_THREADS - 1; k >= 0; --k) {
      const double v = scan[tid][k + 1];
      scan[tid][k + 1] = s;
      s += v;
    }
  }
  __syncthreads();

  // pass 2: forward sweep with running prefixes (and the diagonal term)
  double PA[NL], PB[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    PA[l] = scan[l][tid];
    PB[l] = scan[NL + l][tid];
  }
  for (int p = p0; p < p1; ++p) {
    const double X = p < F.n_rows ? F.a_dev[p] : 0.0;
    const double Y = p < F.n_cols ? F.b_dev[p] : 0.0;
    const double r = F.r_dev[p], inv = 1.0 / r;
    double pw = L0 > 0 ? ipow(r, L0) : 1.0;
    double ip = L0 > 0 ? ipow(inv, L0 + 1) : inv;
    double u = gd * Y * inv, v = gd * X * inv;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      u += g[l] * ip * PB[l];
      v += g[l] * ip * PA[l];
      PA[l] += X * pw;
      PB[l] += Y * pw;
      pw *= r;
      ip *= inv;
    }
    if (p < F.n_rows) F.ga_dev[p] = accumulate ? F.ga_dev[p] + u : u;
    if (p < F.n_cols) F.gb_dev[p] = accumulate ? F.gb_dev[p] + v : v;
  }
  // pass 3: backward sweep with running suffixes (same thread, same elements: no barrier needed)
  double SA[NL], SB[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    SA[l] = scan[2 * NL + l][tid + 1];
    SB[l] = scan[3 * NL + l][tid + 1];
  }
  for (int p = p1 - 1; p >= p0; --p) {
    const double X = p < F.n_rows ? F.a_dev[p] : 0.0;
    const double Y = p < F.n_cols ? F.b_dev[p] : 0.0;
    const double r = F.r_dev[p], inv = 1.0 / r;
    double pw = L0 > 0 ? ipow(r, L0) : 1.0;
    double ip = L0 > 0 ? ipow(inv, L0 + 1) : inv;
    double u = 0.0, v = 0.0;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      u += g[l] * pw * SB[l];
      v += g[l] * pw * SA[l];
      SA[l] += X * ip;
      SB[l] += Y * ip;
      pw *= r;
      ip *= inv;
    }
    if (p < F.n_rows) F.ga_dev[p] += u;
    if (p < F.n_cols) F.gb_dev[p] += v;
  }
}

template <int NL>
int launch(const dwba_form_grad_t* forms, int n, const double* grad, int L0, int n_ltot, const DiagScale& ds,
           int acc, cudaStream_t st) {
  if (cudaFuncSetAttribute(semisep_backward_kernel<NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, BW_SMEM) !=
      cudaSuccess)
    return DWBA_ERR_CUDA;
  // one cluster per form and gradient; the grid's x extent is limited to 2^31 - 1 CTAs
  constexpr int MAX_FORMS = 0x7fffffff / (2 * BW_CLUSTER);
  for (int s0 = 0; s0 < n; s0 += MAX_FORMS) {
    const int m = n - s0 < MAX_FORMS ? n - s0 : MAX_FORMS;
    semisep_backward_kernel<NL><<<m * 2 * BW_CLUSTER, BW_THREADS, BW_SMEM, st>>>(
        forms + s0, grad + (int64_t)s0 * n_ltot, L0, n_ltot, ds, acc, n >= BW_SHORT_FORMS ? BW_SHORT + 1 : 0);
    DWBA_CHECK_LAUNCH();
  }
  if (n >= BW_SHORT_FORMS) {
    semisep_backward_short_kernel<NL><<<n, BW_THREADS, 0, st>>>(forms, grad, L0, n_ltot, ds, acc);
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
  for (int L0 = 0; L0 < n_ltot; L0 += NL_MAX) {
    const int nl = (n_ltot - L0) < NL_MAX ? (n_ltot - L0) : NL_MAX;
    const int rc = launch_nl(nl, forms_dev, n_forms, grad_dev, L0, n_ltot, ds, L0 > 0 ? 1 : 0,
                             (cudaStream_t)stream);
    if (rc != DWBA_OK) return rc;
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
