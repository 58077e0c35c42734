// Direct integrals through the multipole potential of the bound density.
//
// In the reference's Filon direct term (oscillatory_integrals.py:2555-2651) the inner integral
//     int_r2(r_p) = sum_q K_L(r_p, r_q) rho2(r_q) w_q         (:2571, rho2 = u_f u_i)
// depends on the bound states only, so every (l_i, l_f) pair of a transition shares it, and the
// outer sum is a plain weighted dot product with the pair's folded density a (the CC fold of
// chi_f chi_i). Here the inner integral of every multipole is one potential per transition,
//     phi_L(p) = r_p^-(L+1) sum_{q<p} b_q r_q^L + r_p^L sum_{q>p} b_q r_q^-(L+1) + d_L b_p / r_p,
// (K_L is semiseparable; d_L = (1-1e-12)^L is the reference's clamp of the diagonal ratio), built
// exactly in O(N L) with forward prefix and backward suffix sums, and each direct integral is
// I_L = sum_{i<n1} a_i phi_L(i): O(n1 L) per pair instead of an O(n1 L) semiseparable form with
// nine accumulator updates per point and multipole.
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

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

// ---- potentials -------------------------------------------------------------------------------
// A cluster of POT_CLUSTER CTAs takes one potential, each CTA a consecutive share of its points and every
// thread POT_PPT consecutive ones, which its warp holds in shared memory with their radii and inverse
// radii (coalesced on the memory side, consecutive on the thread side). The threads' sums of the prefix
// series b r^L and the suffix series b r^-(L+1) are combined by warp scans, the warps' and then the
// CTAs' totals (each CTA hands its totals to the others through distributed shared memory: one cluster
// barrier), and every row gets
//     phi_L(p) = r_p^-(L+1) (prefix before p) + r_p^L (suffix after p) + d_L b_p / r_p,
// a multipole at a time, written through the warp's shared memory. Up to 16384
// points (with 8 warps per CTA) the operand is read once; longer ones walk their tiles (totals first, then rows; the
// suffix of a tile needs the totals of the tiles after it, which are summed again from the operand).
// About 14 FP64 operations per point and multipole against 8 bytes written: latency for a few potentials,
// the FP64 pipe, barriers and instruction fetch for hundreds. Measured: 4 potentials at N = 15000, L <= 8 in 42 us
// before (CTAs of 1024 rows, each summing all columns outside its rows) and 16 us now; 341 at N = 8000, L <= 10: 197 us
// with eight warps per CTA, of which half had no points, 132 us with four.
namespace cg = cooperative_groups;

constexpr int POT_PPT = 8;               // consecutive points per thread
constexpr int POT_WARP = 32 * POT_PPT;   // points per warp and tile
constexpr int POT_CLUSTER = 8;
constexpr int POT_NW_MAX = 8;            // warps per CTA at most (the launch picks by the longest potential)
constexpr int POT_FEW = 148 * 2 / POT_CLUSTER;  // potentials whose CTAs of eight warps are resident together
constexpr int P_NL = 12;                 // multipoles per launch
// one pad per POT_PPT points: the lanes' runs start in different banks
__device__ __forceinline__ int pot_pos(int i) { return i + i / POT_PPT; }
constexpr int POT_BUF = POT_WARP + POT_WARP / POT_PPT;
constexpr int POT_WARP_SMEM = 4 * POT_BUF * (int)sizeof(double);  // operand, r, 1/r, output of a warp's points

// the two halves of a cluster barrier
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

template <int NL, int POT_NW, bool SPREAD>
__global__ void __cluster_dims__(POT_CLUSTER, 1, 1) __launch_bounds__(32 * POT_NW, 16 / POT_NW)
potential_kernel(const dwba_potential_t* __restrict__ pots, int L0, DiagScale ds) {
  constexpr int PT = 32 * POT_NW;
  constexpr int POT_TILE = PT * POT_PPT;  // points a CTA holds at a time
  constexpr int NS = 2 * NL;  // scanned series: b r^L (prefix), b r^-(L+1) (suffix)
  extern __shared__ double s_buf[];
  __shared__ double s_wtot[NS][POT_NW];
  __shared__ double s_woff[NS][POT_NW];  // the series before (prefix) or after (suffix) each warp's points
  __shared__ double s_all[POT_CLUSTER][NS];
  __shared__ double s_carry[NS];
  cg::cluster_group cluster = cg::this_cluster();
  // another CTA's shared memory may be written once that CTA runs: arrive now (before the descriptor is there, if every
  // CTA stays), wait before the first write
  if (SPREAD) cluster_arrive();
  const int rank = (int)cluster.block_rank();
  const dwba_potential_t D = pots[blockIdx.x / POT_CLUSTER];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = max(D.n_rows, D.n_cols);
  // a potential takes every CTA of its cluster (SPREAD), or as many as it fills with one tile each: the others leave at
  // once (a cluster barrier counts the threads that have not exited)
  const int used = SPREAD ? POT_CLUSTER : min(POT_CLUSTER, max(1, (M + POT_TILE - 1) / POT_TILE));
  if (!SPREAD && rank >= used) return;
  if (!SPREAD) cluster_arrive();
  const int share = ((M + used - 1) / used + POT_WARP - 1) / POT_WARP * POT_WARP;
  const int c0 = min(M, rank * share), c1 = min(M, c0 + share);
  const int n_tiles = (c1 - c0 + POT_TILE - 1) / POT_TILE;
  double* sy = s_buf + warp * 4 * POT_BUF;
  double* sr = sy + POT_BUF;
  double* sv = sr + POT_BUF;
  double* so = sv + POT_BUF;
  const int own = lane * (POT_PPT + 1);
  auto load_tile = [&](int k) -> bool {  // false: the warp has no points in tile k
    const int w0 = c0 + k * POT_TILE + warp * POT_WARP;
    const int left = c1 - w0;
    if (left <= 0) return false;
    double y[POT_PPT], r[POT_PPT];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < POT_PPT; ++j) {
      const int i = j * 32 + lane;
      y[j] = (i < left && w0 + i < D.n_cols) ? D.b_dev[w0 + i] : 0.0;
      r[j] = i < left ? D.r_dev[w0 + i] : 1.0;
    }
#pragma unroll
    for (int j = 0; j < POT_PPT; ++j) {
      const int at = pot_pos(j * 32 + lane);
      sy[at] = y[j];
      sr[at] = r[j];
      sv[at] = 1.0 / r[j];
    }
    __syncwarp();
    return true;
  };
  auto totals = [&](double* t, bool live) {
#pragma unroll
    for (int q = 0; q < NS; ++q) t[q] = 0.0;
    if (!live) return;
#pragma unroll
    for (int j = 0; j < POT_PPT; ++j) {
      const double y = sy[own + j], r = sr[own + j], v = sv[own + j];
      double a = y * (L0 > 0 ? ipow(r, L0) : 1.0), b = y * (L0 > 0 ? ipow(v, L0 + 1) : v);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        t[l] += a;
        t[NL + l] += b;
        a *= r;
        b *= v;
      }
    }
  };
  // exclusive scan of the threads' sums within the warp; the warps' totals go to s_wtot (block-wide)
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
  auto tile_total = [&](int q) {
    double o = 0.0;
#pragma unroll
    for (int w = 0; w < POT_NW; ++w) o += s_wtot[q][w];
    return o;
  };
  // s_woff from the carry and the warps' totals (block-wide)
  auto warp_offsets = [&]() {
    for (int i = tid; i < NS * POT_NW; i += PT) {
      const int q = i / POT_NW, w = i - q * POT_NW;
      double o = s_carry[q];
      if (q < NL) {
        for (int k = 0; k < w; ++k) o += s_wtot[q][k];
      } else {
        for (int k = POT_NW - 1; k > w; --k) o += s_wtot[q][k];
      }
      s_woff[q][w] = o;
    }
    __syncthreads();
  };
  // rows of tile k from the thread's exclusive sums t (warp-wide): both parts of a multipole, then its store
  auto rows = [&](int k, double* t) {
    const int w0 = c0 + k * POT_TILE + warp * POT_WARP;
    double P[POT_PPT], Q[POT_PPT];
#pragma unroll
    for (int j = 0; j < POT_PPT; ++j) {
      const double r = sr[own + j], v = sv[own + j];
      P[j] = L0 > 0 ? ipow(r, L0) : 1.0;
      Q[j] = L0 > 0 ? ipow(v, L0 + 1) : v;
    }
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const double d = ds.v[L0 + l];
      double u[POT_PPT];
      double pre = t[l] + s_woff[l][warp], suf = t[NL + l] + s_woff[NL + l][warp];
#pragma unroll
      for (int j = 0; j < POT_PPT; ++j) {
        const double y = sy[own + j];
        u[j] = fma(Q[j], pre, d * (y * sv[own + j]));
        pre = fma(y, P[j], pre);
      }
#pragma unroll
      for (int j = POT_PPT - 1; j >= 0; --j) {
        u[j] = fma(P[j], suf, u[j]);
        suf = fma(sy[own + j], Q[j], suf);
      }
#pragma unroll
      for (int j = 0; j < POT_PPT; ++j) {
        so[own + j] = u[j];
        P[j] *= sr[own + j];
        Q[j] *= sv[own + j];
      }
      __syncwarp();
      double* phi = D.phi_dev + (int64_t)(L0 + l) * D.stride;
#pragma unroll
      for (int j = 0; j < POT_PPT; ++j) {
        const int p = w0 + j * 32 + lane;
        if (p < c1 && p < D.n_rows) phi[p] = so[pot_pos(j * 32 + lane)];
      }
      __syncwarp();
    }
  };

  // 1. this CTA's totals
  double t[NS];
  bool live = false;
  for (int q = tid; q < NS; q += PT) s_carry[q] = 0.0;
  if (n_tiles == 1) {
    live = load_tile(0);
    totals(t, live);
    scan(t, live);
  } else {
    for (int k = 0; k < n_tiles; ++k) {
      live = load_tile(k);
      totals(t, live);
      scan(t, live);
      for (int q = tid; q < NS; q += PT) s_carry[q] += tile_total(q);
      __syncthreads();
    }
  }
  // 2. handed to every CTA of the cluster, then the parts of the CTAs before and after this one
  __syncthreads();  // s_carry (a CTA without points passed no barrier yet)
  cluster_wait();
  for (int i = tid; i < NS * used; i += PT) {
    const int k = i / NS, q = i - k * NS;
    *cluster.map_shared_rank(&s_all[rank][q], k) = n_tiles == 1 ? tile_total(q) : s_carry[q];
  }
  cluster.sync();
  for (int q = tid; q < NS; q += PT) {
    double o = 0.0;
    if (q < NL) {
      for (int k = 0; k < rank; ++k) o += s_all[k][q];
    } else {
      for (int k = used - 1; k > rank; --k) o += s_all[k][q];
    }
    s_carry[q] = o;
  }
  __syncthreads();
  // 3. the rows
  if (n_tiles == 1) {
    warp_offsets();
    if (live) rows(0, t);
    return;
  }
  for (int k = 0; k < n_tiles; ++k) {
    // suffix over the CTA's later tiles, from the operand (tiles in descending order, as the carries)
    double* s_suf = s_all[0];  // free after the barrier above
    double* s_keep = s_all[1];
    for (int q = tid; q < NS; q += PT) s_suf[q] = s_keep[q] = s_carry[q];
    __syncthreads();
    for (int m = n_tiles - 1; m > k; --m) {
      live = load_tile(m);
      totals(t, live);
      scan(t, live);
      for (int q = NL + tid; q < NS; q += PT) s_suf[q] += tile_total(q);
      __syncthreads();
    }
    live = load_tile(k);
    totals(t, live);
    scan(t, live);
    for (int q = tid; q < NS; q += PT) s_carry[q] = s_suf[q];
    __syncthreads();
    warp_offsets();
    if (live) rows(k, t);
    __syncthreads();
    for (int q = tid; q < NS; q += PT) s_carry[q] = q < NL ? s_keep[q] + tile_total(q) : s_keep[q];
    __syncthreads();
  }
}

template <int NL, int NW, bool SPREAD = true>
int launch_pot_nw(const dwba_potential_t* pots, int n, int L0, const DiagScale& ds, cudaStream_t st) {
  constexpr int SMEM = NW * POT_WARP_SMEM;
  if (cudaFuncSetAttribute(potential_kernel<NL, NW, SPREAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) !=
      cudaSuccess)
    return DWBA_ERR_CUDA;
  constexpr int MAX_POTS = 0x7fffffff / POT_CLUSTER;  // one cluster per potential
  for (int s0 = 0; s0 < n; s0 += MAX_POTS) {
    const int m = (n - s0) < MAX_POTS ? (n - s0) : MAX_POTS;
    potential_kernel<NL, NW, SPREAD><<<m * POT_CLUSTER, 32 * NW, SMEM, st>>>(pots + s0, L0, ds);
    DWBA_CHECK_LAUNCH();
  }
  return DWBA_OK;
}

template <int NL>
int launch_pot(const dwba_potential_t* pots, int n, int max_len, int L0, const DiagScale& ds, cudaStream_t st) {
  // More than the GPU holds at once, lengths unknown: four warps per CTA, and a potential takes the CTAs it fills. 300
  // potentials, L <= 8: N = 2000 37 us (122 us with eight warps and the whole cluster each), N = 8000 91 us (141 us),
  // but N = 15000, two tiles per CTA, 320 us (176 us).
  if (max_len == 0x7fffffff && n > POT_FEW) return launch_pot_nw<NL, 4, false>(pots, n, L0, ds, st);
  // as many warps as the longest potential needs for one tile per CTA: warps without points would only
  // take registers from live ones
  const int runs = (int)(((int64_t)max_len + POT_CLUSTER * POT_WARP - 1) / (POT_CLUSTER * POT_WARP));
  if (runs <= 1) return launch_pot_nw<NL, 1>(pots, n, L0, ds, st);
  if (runs <= 2) return launch_pot_nw<NL, 2>(pots, n, L0, ds, st);
  if (runs <= 4) return launch_pot_nw<NL, 4>(pots, n, L0, ds, st);
  return launch_pot_nw<NL, POT_NW_MAX>(pots, n, L0, ds, st);
}

int launch_pot_nl(int nl, const dwba_potential_t* pots, int n, int max_len, int L0, const DiagScale& ds,
                  cudaStream_t st) {
  switch (nl) {
#define DWBA_CASE(N) \
  case N: return launch_pot<N>(pots, n, max_len, L0, ds, st);
    DWBA_CASE(1) DWBA_CASE(2) DWBA_CASE(3) DWBA_CASE(4) DWBA_CASE(5) DWBA_CASE(6) DWBA_CASE(7) DWBA_CASE(8)
    DWBA_CASE(9) DWBA_CASE(10) DWBA_CASE(11) DWBA_CASE(12)
#undef DWBA_CASE
    default: return DWBA_ERR_INVALID_ARG;
  }
}

// ---- dot forms --------------------------------------------------------------------------------
// A CTA takes DOT_PER_CTA consecutive descriptors that share one potential (the caller groups
// them and pads a group with empty descriptors, n_rows = 0). Tiles of the potential's rows
// (NL multipoles x DOT_TILE points) are staged in shared memory once for all of them, in two
// buffers: the loads of tile t+1 (potential and the descriptors' rows) are issued into registers
// before tile t is accumulated, so each tile costs one barrier and no exposed load latency. Warp
// w accumulates descriptors 2w and 2w+1 (each staged value serves two pairs), lanes stride over
// the tile's points, and the lanes' sums are added by shuffles in a fixed order.
constexpr int DOT_THREADS = 256;
constexpr int DOT_PER_CTA = 16;
constexpr int DOT_TILE = 128;
constexpr int DOT_NL = 16;
constexpr int DOT_RPL = DOT_TILE / 32;  // rows per lane and tile

template <int NL>
__global__ void __launch_bounds__(DOT_THREADS)
dot_kernel(const dwba_dot_t* __restrict__ dots, int n, int L0, int n_ltot) {
  constexpr int PER = (NL * DOT_TILE + DOT_THREADS - 1) / DOT_THREADS;  // staged values per thread
  __shared__ double sphi[2][NL * DOT_TILE];
  __shared__ int s_rows;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int d0 = blockIdx.x * DOT_PER_CTA;
  const int da = d0 + 2 * warp, db = da + 1;
  const dwba_dot_t A = da < n ? dots[da] : dwba_dot_t{nullptr, nullptr, nullptr, 0, 0};
  const dwba_dot_t B = db < n ? dots[db] : dwba_dot_t{nullptr, nullptr, nullptr, 0, 0};
  if (tid == 0) s_rows = 0;
  __syncthreads();
  if (lane == 0) atomicMax(&s_rows, max(A.n_rows, B.n_rows));
  __syncthreads();
  const int rows = s_rows;
  const int n_tiles = (rows + DOT_TILE - 1) / DOT_TILE;
  // the group's potential: the first descriptor's (every non-empty one of the group shares it)
  const dwba_dot_t G = dots[d0];
  double pf[PER], xa[DOT_RPL], xb[DOT_RPL];
  auto load_tile = [&](int i0) {
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int k = tid + m * DOT_THREADS;
      const int l = k / DOT_TILE, i = i0 + (k - l * DOT_TILE);
      pf[m] = (k < NL * DOT_TILE && i < rows) ? G.phi_dev[(int64_t)(L0 + l) * G.stride + i] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < DOT_RPL; ++q) {
      const int i = i0 + q * 32 + lane;
      xa[q] = i < A.n_rows ? A.a_dev[i] : 0.0;
      xb[q] = i < B.n_rows ? B.a_dev[i] : 0.0;
    }
  };
  double acc_a[NL], acc_b[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) acc_a[l] = acc_b[l] = 0.0;
  if (n_tiles > 0) load_tile(0);
  for (int t = 0; t < n_tiles; ++t) {
    double* buf = sphi[t & 1];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int k = tid + m * DOT_THREADS;
      if (k < NL * DOT_TILE) buf[k] = pf[m];
    }
    double ca[DOT_RPL], cb[DOT_RPL];
#pragma unroll
    for (int q = 0; q < DOT_RPL; ++q) {
      ca[q] = xa[q];
      cb[q] = xb[q];
    }
    // one barrier per tile: it publishes this buffer, and every thread passed the previous one
    // only after accumulating the tile that last used this buffer
    __syncthreads();
    if (t + 1 < n_tiles) load_tile((t + 1) * DOT_TILE);  // in flight during the accumulation
#pragma unroll
    for (int q = 0; q < DOT_RPL; ++q) {
      const int ii = q * 32 + lane;
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        const double ph = buf[l * DOT_TILE + ii];
        acc_a[l] = fma(ca[q], ph, acc_a[l]);
        acc_b[l] = fma(cb[q], ph, acc_b[l]);
      }
    }
  }
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    double va = acc_a[l], vb = acc_b[l];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      va += __shfl_down_sync(0xffffffffu, va, off);
      vb += __shfl_down_sync(0xffffffffu, vb, off);
    }
    if (lane == 0) {
      if (A.out_dev != nullptr) A.out_dev[L0 + l] = va;
      if (B.out_dev != nullptr) B.out_dev[L0 + l] = vb;
    }
  }
}

template <int NL>
int launch_dot(const dwba_dot_t* dots, int n, int L0, int n_ltot, cudaStream_t st) {
  const int grid = (n + DOT_PER_CTA - 1) / DOT_PER_CTA;
  dot_kernel<NL><<<grid, DOT_THREADS, 0, st>>>(dots, n, L0, n_ltot);
  DWBA_CHECK_LAUNCH();
  return DWBA_OK;
}

int launch_dot_nl(int nl, const dwba_dot_t* dots, int n, int L0, int n_ltot, cudaStream_t st) {
  switch (nl) {
#define DWBA_CASE(N) \
  case N: return launch_dot<N>(dots, n, L0, n_ltot, st);
    DWBA_CASE(1) DWBA_CASE(2) DWBA_CASE(3) DWBA_CASE(4) DWBA_CASE(5) DWBA_CASE(6) DWBA_CASE(7) DWBA_CASE(8)
    DWBA_CASE(9) DWBA_CASE(10) DWBA_CASE(11) DWBA_CASE(12) DWBA_CASE(13) DWBA_CASE(14) DWBA_CASE(15)
    DWBA_CASE(16)
#undef DWBA_CASE
    default: return DWBA_ERR_INVALID_ARG;
  }
}

}  // namespace

extern "C" int dwba_multipole_potentials_sized(const dwba_potential_t* pots_dev, int n, int max_len, int L_max,
                                               const double* diag_scale_host, double r_min_all, double r_max_all,
                                               dwba_stream_t stream) {
  if (n <= 0) return DWBA_OK;
  if (!pots_dev || !diag_scale_host || L_max < 0 || L_max > DWBA_MAX_L || !(r_min_all > 0.0) ||
      !(r_max_all >= r_min_all) || max_len < 0)
    return DWBA_ERR_INVALID_ARG;
  // r^L and r^-(L+1) must stay finite and normal in FP64
  const double lmin = log10(r_min_all), lmax = log10(r_max_all);
  if (fmax(fabs(lmin), fabs(lmax)) * (L_max + 1) > 280.0) return DWBA_ERR_UNSUPPORTED;
  DiagScale ds;
  for (int l = 0; l <= DWBA_MAX_L; ++l) ds.v[l] = l <= L_max ? diag_scale_host[l] : 0.0;
  const int n_ltot = L_max + 1;
  for (int L0 = 0; L0 < n_ltot; L0 += P_NL) {
    const int nl = (n_ltot - L0) < P_NL ? (n_ltot - L0) : P_NL;
    const int rc = launch_pot_nl(nl, pots_dev, n, max_len, L0, ds, (cudaStream_t)stream);
    if (rc != DWBA_OK) return rc;
  }
  return DWBA_OK;
}

extern "C" int dwba_multipole_potentials(const dwba_potential_t* pots_dev, int n, int L_max,
                                         const double* diag_scale_host, double r_min_all, double r_max_all,
                                         dwba_stream_t stream) {
  return dwba_multipole_potentials_sized(pots_dev, n, 0x7fffffff, L_max, diag_scale_host, r_min_all, r_max_all, stream);
}

extern "C" int dwba_dot_forms(const dwba_dot_t* dots_dev, int n, int L_max, dwba_stream_t stream) {
  if (n <= 0) return DWBA_OK;
  if (!dots_dev || L_max < 0 || L_max > DWBA_MAX_L) return DWBA_ERR_INVALID_ARG;
  const int n_ltot = L_max + 1;
  for (int L0 = 0; L0 < n_ltot; L0 += DOT_NL) {
    const int nl = (n_ltot - L0) < DOT_NL ? (n_ltot - L0) : DOT_NL;
    const int rc = launch_dot_nl(nl, dots_dev, n, L0, n_ltot, (cudaStream_t)stream);
    if (rc != DWBA_OK) return rc;
  }
  return DWBA_OK;
}
