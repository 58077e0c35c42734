// Amplitudes, DCS and TCS from the radial integrals of many partial-wave channels.
//
// Per target sublevel pair a and channel p the amplitudes are linear in the integrals with one
// spherical harmonic of l_f as angular factor (dwba_coupling.py:285-505):
//   f_a(theta) = sum_p yd[a][p](theta) sum_L cf[a][p][L] I_dir[p][L]
//   g_a(theta) = sum_p ye[a][p](theta) sum_L cg[a][p][L] I_exc[p][L]
// and DCS(theta) = pref sum_a [1/4 |f_a + g_a|^2 + 3/4 |f_a - g_a|^2], clipped at 0
// (sigma_total.py:147-177); TCS = 2 pi trapz(sin(theta) DCS, theta) (sigma_total.py:179-217).
// The coefficients and the Y tables are read once (8 MB for 840 channels, three sublevel pairs and 181
// angles), so the kernel is bound by latency: a cluster of DCS_CLUSTER CTAs takes DCS_ANGLES angles, its
// CTAs and their warps share the channels, and the partial amplitudes meet in shared memory (one CTA's
// warps, then the cluster's CTAs through distributed shared memory, both in a fixed order). No scratch
// buffer and no second launch is needed. The trapezoid runs in a fixed tree.
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int DCS_THREADS = 512;
constexpr int DCS_WARPS = DCS_THREADS / 32;
constexpr int DCS_ANGLES = 32;   // one per lane: a warp reads 256 contiguous bytes of a Y row
constexpr int DCS_CLUSTER = 8;
constexpr int DCS_PC = 256;      // channels whose multipole sums a CTA stages at a time

// (181 angles, 840 channels, three sublevel pairs, L <= 6: the whole call 22 us, its host side included;
// one thread per angle over all channels, in two CTAs, took 3041 us for this kernel alone.)
__global__ void __cluster_dims__(DCS_CLUSTER, 1, 1) __launch_bounds__(DCS_THREADS)
dcs_kernel(const double2* __restrict__ cf, const double2* __restrict__ cg_,
           const double* __restrict__ yd, const double* __restrict__ ye,
           const double* __restrict__ I_dir, const double* __restrict__ I_exc, int n_M, int P,
           int nl, int n_theta, double pref, double* __restrict__ dcs) {
  __shared__ double s_mul[4][DCS_PC];                     // multipole sums of the staged channels
  __shared__ double s_red[DCS_WARPS][4][DCS_ANGLES];      // per warp: f and g (re, im)
  __shared__ double s_part[2][4][DCS_ANGLES];             // per CTA, double-buffered over sublevel pairs
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = (blockIdx.x / DCS_CLUSTER) * DCS_ANGLES + lane;
  const bool in = t < n_theta;
  const int per = (P + DCS_CLUSTER - 1) / DCS_CLUSTER;
  const int p_lo = min(P, rank * per), p_hi = min(P, p_lo + per);
  double acc = 0.0;  // rank 0, warp 0
  for (int a = 0; a < n_M; ++a) {
    double f[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c0 = p_lo; c0 < p_hi; c0 += DCS_PC) {
      const int nc = min(DCS_PC, p_hi - c0);
      __syncthreads();  // the previous chunk's sums are consumed
      for (int k = tid; k < 2 * nc; k += DCS_THREADS) {  // direct sums of the chunk, then exchange sums
        const int p = k < nc ? k : k - nc, kind = k < nc ? 0 : 1;
        const double2* c = (kind ? cg_ : cf) + ((int64_t)a * P + c0 + p) * nl;
        const double* I = (kind ? I_exc : I_dir) + (int64_t)(c0 + p) * nl;
        double re = 0.0, im = 0.0;
        for (int L = 0; L < nl; ++L) {
          const double2 v = c[L];
          re += v.x * I[L];
          im += v.y * I[L];
        }
        s_mul[2 * kind][p] = re;
        s_mul[2 * kind + 1][p] = im;
      }
      __syncthreads();
      if (in) {
#pragma unroll 4
        for (int p = warp; p < nc; p += DCS_WARPS) {
          const int64_t row = ((int64_t)a * P + c0 + p) * n_theta + t;
          const double y1 = yd[row], y2 = ye[row];
          f[0] += y1 * s_mul[0][p];
          f[1] += y1 * s_mul[1][p];
          f[2] += y2 * s_mul[2][p];
          f[3] += y2 * s_mul[3][p];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) s_red[warp][q][lane] = f[q];
    __syncthreads();
    if (warp < 4) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < DCS_WARPS; ++w) v += s_red[w][warp][lane];
      s_part[a & 1][warp][lane] = v;
    }
    // publishes this pair's partial sums; the buffer is written again two pairs later, after the next
    // barrier, which rank 0 reaches only once it has read it
    cluster.sync();
    if (rank == 0 && warp == 0) {
      double g[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double v = 0.0;
        for (int k = 0; k < DCS_CLUSTER; ++k) v += *cluster.map_shared_rank(&s_part[a & 1][q][lane], k);
        g[q] = v;
      }
      const double sr = g[0] + g[2], si = g[1] + g[3], dr = g[0] - g[2], di = g[1] - g[3];
      acc += pref * (0.25 * (sr * sr + si * si) + 0.75 * (dr * dr + di * di));
    }
  }
  if (rank == 0 && warp == 0 && in) dcs[t] = acc > 0.0 ? acc : 0.0;
  cluster.sync();  // no CTA leaves while its shared memory may still be read
}

// Few channels and many angles: one thread per angle over all channels. A cluster has nothing to share then: its eight
// CTAs and their barriers cost about 3.5 ns per angle and sublevel pair, a thread's serial sum about 1.1 us per channel
// and sublevel pair, so the line is drawn at DCS_FEW angles per channel (one pair: 1 channel and 3000 angles 24 us by
// clusters and 16 us by threads, 20 channels and 20000 angles 123 and 81 us; 10 and 3000: 25 and 27 us; 80 and 20000:
// 125 and 155 us).
constexpr int DCS_FEW = 320;

__global__ void dcs_angles_kernel(const double2* __restrict__ cf, const double2* __restrict__ cg_,
                                  const double* __restrict__ yd, const double* __restrict__ ye,
                                  const double* __restrict__ I_dir, const double* __restrict__ I_exc, int n_M, int P,
                                  int nl, int n_theta, double pref, double* __restrict__ dcs) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_theta; t += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int a = 0; a < n_M; ++a) {
      double f[4] = {0.0, 0.0, 0.0, 0.0};  // f and g (re, im)
      for (int p = 0; p < P; ++p) {
        const int64_t row = (int64_t)a * P + p;
        const double y[2] = {yd[row * n_theta + t], ye[row * n_theta + t]};
#pragma unroll
        for (int kind = 0; kind < 2; ++kind) {
          const double2* c = (kind ? cg_ : cf) + row * nl;
          const double* I = (kind ? I_exc : I_dir) + (int64_t)p * nl;
          double re = 0.0, im = 0.0;
          for (int L = 0; L < nl; ++L) {
            const double2 v = c[L];
            re += v.x * I[L];
            im += v.y * I[L];
          }
          f[2 * kind] += y[kind] * re;
          f[2 * kind + 1] += y[kind] * im;
        }
      }
      const double sr = f[0] + f[2], si = f[1] + f[3], dr = f[0] - f[2], di = f[1] - f[3];
      acc += pref * (0.25 * (sr * sr + si * si) + 0.75 * (dr * dr + di * di));
    }
    dcs[t] = acc > 0.0 ? acc : 0.0;
  }
}

// 2 pi sum of trapezoids of sin(theta) DCS, one block, fixed reduction tree
__global__ void tcs_kernel(const double* __restrict__ theta, const double* __restrict__ dcs, int n, double* tcs) {
  __shared__ double red[256];
  double s = 0.0;
  for (int i = threadIdx.x; i + 1 < n; i += blockDim.x)
    s += 0.5 * (theta[i + 1] - theta[i]) * (sin(theta[i]) * dcs[i] + sin(theta[i + 1]) * dcs[i + 1]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *tcs = 2.0 * M_PI * red[0];
}

}  // namespace

extern "C" int dwba_cross_sections(const double* cf_dev, const double* cg_dev, const double* yd_dev,
                                   const double* ye_dev, const double* I_dir_dev, const double* I_exc_dev,
                                   const double* theta_dev, int n_M, int P, int nl, int n_theta, double pref,
                                   double* dcs_dev, double* tcs_dev, dwba_stream_t stream) {
  if (n_theta <= 0) return DWBA_OK;
  if (!cf_dev || !cg_dev || !yd_dev || !ye_dev || !I_dir_dev || !I_exc_dev || !theta_dev || !dcs_dev || n_M < 1 ||
      P < 0 || nl < 1 || nl > DWBA_MAX_L + 1)
    return DWBA_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if ((int64_t)P * DCS_FEW < n_theta) {
    dcs_angles_kernel<<<dwba_grid_1d(n_theta, 128), 128, 0, st>>>((const double2*)cf_dev, (const double2*)cg_dev, yd_dev,
                                                                  ye_dev, I_dir_dev, I_exc_dev, n_M, P, nl, n_theta,
                                                                  pref, dcs_dev);
  } else {
    const int blocks = dwba_grid_1d(n_theta, DCS_ANGLES, (1 << 30) / DCS_CLUSTER) * DCS_CLUSTER;
    dcs_kernel<<<blocks, DCS_THREADS, 0, st>>>((const double2*)cf_dev, (const double2*)cg_dev, yd_dev, ye_dev, I_dir_dev,
                                               I_exc_dev, n_M, P, nl, n_theta, pref, dcs_dev);
  }
  DWBA_CHECK_LAUNCH();
  if (tcs_dev) {
    tcs_kernel<<<1, 256, 0, st>>>(theta_dev, dcs_dev, n_theta, tcs_dev);
    DWBA_CHECK_LAUNCH();
  }
  return DWBA_OK;
}
