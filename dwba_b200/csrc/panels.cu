// Panels: the integrals of many pairs that share their operands, as FP64 matrix products.
//
// All pairs of an energy point share their node set, so the folded exchange operands depend on one wave each
// (a = T (u_f chi_i) on l_i, b = B (chi_f u_i) on l_f) and the direct density's fold can be moved to the other
// side (T is symmetric: (T chi_f chi_i)^T phi_L = sum_x chi_i chi_f psi_L, psi_L = T phi_L). With the potentials
// Phi_{f,L} = K_L b_f of the distinct b (dwba_multipole_potentials),
//     exchange  I_L[i, f] = sum_x a_i[x] Phi_{f,L}[x],      direct  I_L[i, f] = sum_x chi_i[x] (chi_f[x] psi_L[x]),
// both a product of M rows with F column blocks of L_max + 1 columns (dwba_matrix_elements.py:1113-1116 and
// oscillatory_integrals.py:2609-2644, :2745-2770 contract one pair and multipole at a time).
//
// A CTA takes 64 rows x 64 columns x one chunk of the grid on the FP64 tensor pipe (mma.m8n8k4, products and sums
// in FP64); the chunks' partial tiles are added in a fixed order by a second kernel. The chunk length depends on
// the panel's own grid alone, so a panel's results do not depend on what else is launched with it.
#include <algorithm>
#include <new>
#include <utility>
#include <vector>

#include "common.cuh"

namespace {

constexpr int PM = 64;           // rows per CTA
constexpr int PN = 64;           // columns per CTA
constexpr int PK = 16;           // grid points per step
constexpr int P_THREADS = 128;   // 4 warps, each 64 rows x 16 columns
static_assert(P_THREADS == PM + PN, "one thread per row and column pointer");
constexpr int P_LD = PK + 4;     // shared-memory row: 4 mod 16 doubles, so a fragment's rows fall in different banks
constexpr int P_CHUNK_MIN = 256;
constexpr int P_CHUNKS = 16;     // chunks per panel at most (longer grids have longer chunks)

__host__ __device__ inline int panel_chunk(int n) {
  int c = (n + P_CHUNKS - 1) / P_CHUNKS;
  c = (c + PK - 1) / PK * PK;
  return c < P_CHUNK_MIN ? P_CHUNK_MIN : c;
}
__host__ __device__ inline int panel_chunks(int n) {
  const int c = panel_chunk(n);
  return n > 0 ? (n + c - 1) / c : 1;
}

__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

struct PanelShared {
  double A[2][PM * P_LD], B[2][PN * P_LD];
  const double* row[PM];
  const double* phi[PN];
  const double* mul[PN];
};

// The chunk's product for MT 8-row tiles (a compile-time count: a predicated-off mma still takes its slot on
// the tensor pipe). MUL: the columns have a second factor.
template <int MT, bool MUL>
__device__ __forceinline__ void panel_tile(PanelShared& S, int k0, int k1, int mr, int nc, double* __restrict__ out,
                                           int N) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // loader: point tid % 16 of rows / columns tid / 16 + 8 q
  const int lk = tid & (PK - 1), lr = tid / PK;
  double ra[MT], rb[PN / 8], rm[PN / 8];
  auto load = [&](int k) {
    const int x = k + lk;
    const bool in = x < k1;
#pragma unroll
    for (int q = 0; q < MT; ++q) {
      const int m = lr + 8 * q;
      ra[q] = (in && m < mr) ? __ldg(S.row[m] + x) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < PN / 8; ++q) {
      const int c = lr + 8 * q;
      const bool ok = in && c < nc;
      rb[q] = ok ? __ldg(S.phi[c] + x) : 0.0;
      if (MUL) rm[q] = ok ? __ldg(S.mul[c] + x) : 0.0;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < MT; ++q) S.A[buf][(lr + 8 * q) * P_LD + lk] = ra[q];
#pragma unroll
    for (int q = 0; q < PN / 8; ++q) S.B[buf][(lr + 8 * q) * P_LD + lk] = MUL ? rb[q] * rm[q] : rb[q];
  };
  double acc[MT][2][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int fr = lane >> 2, fk = lane & 3;
  const bool live = warp * 16 < nc;  // the warp has columns
  load(k0);
  int buf = 0;
  for (int k = k0; k < k1; k += PK) {
    store(buf);
    __syncthreads();  // publishes this buffer; the other one was consumed before the previous barrier
    if (k + PK < k1) load(k + PK);
    if (live) {
      const double* sa = S.A[buf] + fr * P_LD + fk;
      const double* sb = S.B[buf] + (warp * 16 + fr) * P_LD + fk;
#pragma unroll
      for (int kk = 0; kk < PK; kk += 4) {
        const double b0 = sb[kk], b1 = sb[8 * P_LD + kk];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const double a = sa[8 * i * P_LD + kk];
          mma_f64(acc[i][0][0], acc[i][0][1], a, b0);
          mma_f64(acc[i][1][0], acc[i][1][1], a, b1);
        }
      }
    }
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int m = 8 * i + fr;
    if (m >= mr) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = warp * 16 + 8 * j + 2 * fk + h;
        if (c < nc) out[(int64_t)m * N + c] = acc[i][j][h];
      }
    }
  }
}

__global__ void __launch_bounds__(P_THREADS, 3)
panel_kernel(const dwba_panel_t* __restrict__ panels, const dwba_panel_cta_t* __restrict__ ctas, int nl,
             double* __restrict__ partial) {
  __shared__ PanelShared S;
  const dwba_panel_cta_t C = ctas[blockIdx.x];
  const dwba_panel_t P = panels[C.panel];
  const int m0 = C.m_tile * PM, n0 = C.n_tile * PN;
  const int N = P.F * nl;
  const int mr = min(PM, P.M - m0), nc = min(PN, N - n0);
  const int chunk = panel_chunk(P.n);
  const int k0 = C.chunk * chunk, k1 = min(P.n, k0 + chunk);
  const int tid = threadIdx.x;
  if (tid < PM) {
    S.row[tid] = tid < mr ? P.rows_dev[m0 + tid] : nullptr;
  } else {
    const int c = tid - PM;
    const double *phi = nullptr, *mul = nullptr;
    if (c < nc) {
      const int f = (n0 + c) / nl, l = n0 + c - f * nl;
      const dwba_panel_col_t d = P.cols_dev[f];
      phi = d.phi_dev + (int64_t)l * P.stride;
      mul = d.mul_dev;
    }
    S.phi[c] = phi;
    S.mul[c] = mul;
  }
  __syncthreads();
  double* out = partial + P.part_off + (int64_t)C.chunk * P.M * N + (int64_t)m0 * N + n0;
  const bool has_mul = S.mul[0] != nullptr;  // the same for every column of a panel
  switch ((mr + 7) / 8) {
#define DWBA_CASE(MT)                                                       \
  case MT:                                                                  \
    if (has_mul) panel_tile<MT, true>(S, k0, k1, mr, nc, out, N);           \
    else panel_tile<MT, false>(S, k0, k1, mr, nc, out, N);                  \
    break;
    DWBA_CASE(1) DWBA_CASE(2) DWBA_CASE(3) DWBA_CASE(4) DWBA_CASE(5) DWBA_CASE(6) DWBA_CASE(7) DWBA_CASE(8)
#undef DWBA_CASE
    default: break;
  }
}

__global__ void panel_reduce_kernel(const dwba_panel_t* __restrict__ panels, int nl, const double* __restrict__ partial) {
  const dwba_panel_t P = panels[blockIdx.y];
  const int N = P.F * nl, nk = panel_chunks(P.n);
  const int64_t total = (int64_t)P.M * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int m = (int)(i / N), c = (int)(i - (int64_t)m * N);
    const int f = c / nl, l = c - f * nl;
    double* out = P.out_dev[(int64_t)m * P.F + f];
    if (!out) continue;
    const double* src = partial + P.part_off + i;
    double s = 0.0;
    for (int k = 0; k < nk; ++k) s += src[k * total];
    out[l] = s;
  }
}

}  // namespace

extern "C" int64_t dwba_panel_plan(dwba_panel_t* panels_host, int n_panels, int L_max, dwba_panel_cta_t* ctas_host,
                                   int64_t* n_partial) {
  if (n_panels < 0 || (n_panels > 0 && !panels_host) || L_max < 0 || L_max > DWBA_MAX_L || !n_partial) return -1;
  int64_t n_cta = 0, part = 0;
  for (int p = 0; p < n_panels; ++p) {
    dwba_panel_t& P = panels_host[p];
    if (P.M < 0 || P.F < 0 || P.n < 0 || P.stride < P.n) return -1;
    const int64_t N = (int64_t)P.F * (L_max + 1);
    if (N > 0x7fffffffLL) return -1;
    const int mt = (P.M + PM - 1) / PM, nt = (int)((N + PN - 1) / PN), nk = panel_chunks(P.n);
    P.part_off = part;
    part += (int64_t)nk * P.M * N;
    if (ctas_host) {
      dwba_panel_cta_t* o = ctas_host + n_cta;
      for (int k = 0; k < nk; ++k)
        for (int b = 0; b < nt; ++b)
          for (int a = 0; a < mt; ++a) *o++ = dwba_panel_cta_t{p, a, b, k};
    }
    n_cta += (int64_t)nk * nt * mt;
  }
  *n_partial = part;
  return n_cta;
}

// ---- host: which entries share their operands ---------------------------------------------------
namespace {

// small numbers for the distinct values of an array, in order of first use
struct Ids {
  std::vector<int32_t> of, back;
  explicit Ids(size_t n) : of(n, -1) {}
  int32_t get(int64_t v) {
    if (of[v] < 0) {
      of[v] = (int32_t)back.size();
      back.push_back((int32_t)v);
    }
    return of[v];
  }
  void clear() {
    for (int32_t v : back) of[v] = -1;
    back.clear();
  }
};

uint64_t mix(uint64_t x) {  // splitmix64
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Panels of the combinations (row[e], col[e]), each at most once: columns used with the same set of rows go
// together, so every panel is complete. Appends M, F, the rows, the columns and the entry of every
// combination; false when a combination is repeated (or a signature collides).
struct Panels {
  std::vector<int32_t> M, F, rows, cols, entry;
};
bool split_panels(const std::vector<int32_t>& row, const std::vector<int32_t>& col, int nr, int nc,
                  const int32_t* entry_of, Panels& out) {
  struct Sig {
    uint64_t h;
    int32_t n, c;
  };
  std::vector<Sig> sig(nc);
  for (int c = 0; c < nc; ++c) sig[c] = Sig{0, 0, c};
  for (size_t e = 0; e < row.size(); ++e) {
    sig[col[e]].h += mix((uint64_t)row[e]);
    ++sig[col[e]].n;
  }
  std::stable_sort(sig.begin(), sig.end(), [](const Sig& a, const Sig& b) { return a.h != b.h ? a.h < b.h : a.n < b.n; });
  std::vector<int32_t> group(nc), at(nc), first;  // group of a column and its position there
  int ng = 0;
  std::vector<int32_t> gF, gM;
  for (int i = 0; i < nc; ++i) {
    if (i == 0 || sig[i].h != sig[i - 1].h || sig[i].n != sig[i - 1].n) {
      ++ng;
      gF.push_back(0);
      gM.push_back(sig[i].n);
    }
    group[sig[i].c] = ng - 1;
    at[sig[i].c] = gF[ng - 1]++;
  }
  std::vector<std::vector<int32_t>> by(ng);
  for (size_t e = 0; e < row.size(); ++e) by[group[col[e]]].push_back((int32_t)e);
  std::vector<int32_t> pos(nr, -1);
  for (int g = 0; g < ng; ++g) {
    const int M = gM[g], F = gF[g];
    const size_t base = out.entry.size(), r0 = out.rows.size(), c0 = out.cols.size();
    out.entry.resize(base + (size_t)M * F, -1);
    out.cols.resize(c0 + F);
    int m = 0;
    for (int32_t e : by[g]) {
      if (pos[row[e]] < 0) {
        if (m == M) return false;  // more rows than a column has: the signatures collided
        pos[row[e]] = m++;
        out.rows.push_back(row[e]);
      }
      int32_t& slot = out.entry[base + (size_t)pos[row[e]] * F + at[col[e]]];
      if (slot >= 0) return false;  // repeated combination
      slot = entry_of[e];
      out.cols[c0 + at[col[e]]] = col[e];
    }
    if (m != M || by[g].size() != (size_t)M * F) return false;
    for (size_t i = r0; i < out.rows.size(); ++i) pos[out.rows[i]] = -1;
    out.M.push_back(M);
    out.F.push_back(F);
  }
  return true;
}

}  // namespace

extern "C" int dwba_panel_layout(const dwba_panel_entry_t* entries, int n, int n_sets, int n_rows, int n_trans,
                                 double min_share, int min_forms, dwba_panel_layout_t* out) {
  if (n < 0 || n_sets < 0 || n_rows < 1 || n_trans < 1 || !out || (n > 0 && !entries)) return DWBA_ERR_INVALID_ARG;
  out->n_a = out->n_b = out->n_psi = out->n_direct = out->n_exchange = 0;
  try {
    std::vector<std::vector<int32_t>> by(n_sets);
    for (int e = 0; e < n; ++e) {
      const dwba_panel_entry_t& E = entries[e];
      if (E.set < 0 || E.set >= n_sets || E.t < 0 || E.t >= n_trans || E.w_i < 0 || E.w_i >= n_rows || E.w_f < 0 ||
          E.w_f >= n_rows || E.u_i < 0 || E.u_i >= n_rows || E.u_f < 0 || E.u_f >= n_rows)
        return DWBA_ERR_INVALID_ARG;
      out->ia[e] = out->ib[e] = -1;
      by[E.set].push_back(e);
    }
    Ids u(n_rows), w(n_rows), tt(n_trans), wr(n_rows);
    int64_t d_rows = 0, d_cols = 0, d_ent = 0, x_rows = 0, x_cols = 0, x_ent = 0;
    for (int k = 0; k < n_sets; ++k) {
      const std::vector<int32_t>& E = by[k];
      const size_t m = E.size();
      if (m < (size_t)min_forms || m < 1) continue;
      std::vector<int32_t> ia(m), ib(m), ir(m), ic(m);
      // operands numbered wave by wave (those of one wave together), functions in order of first use
      struct Items {
        std::vector<int32_t> u, w;
      } A, B;
      auto number = [&](bool first, std::vector<int32_t>& id, Items& it) {
        u.clear();
        w.clear();
        for (int32_t e : E) {
          u.get(first ? entries[e].u_f : entries[e].u_i);
          w.get(first ? entries[e].w_i : entries[e].w_f);
        }
        const size_t nu = u.back.size(), nw = w.back.size();
        std::vector<int32_t> tab(nu * nw, -1);
        for (int32_t e : E)
          tab[(size_t)w.get(first ? entries[e].w_i : entries[e].w_f) * nu + u.get(first ? entries[e].u_f : entries[e].u_i)] = 0;
        for (size_t q = 0; q < tab.size(); ++q)
          if (tab[q] == 0) {
            tab[q] = (int32_t)it.u.size();
            it.u.push_back(u.back[q % nu]);
            it.w.push_back(w.back[q / nu]);
          }
        for (size_t i = 0; i < m; ++i) {
          const dwba_panel_entry_t& x = entries[E[i]];
          id[i] = tab[(size_t)w.get(first ? x.w_i : x.w_f) * nu + u.get(first ? x.u_f : x.u_i)];
        }
      };
      number(false, ib, B);
      if ((double)m < min_share * (double)B.u.size()) continue;
      number(true, ia, A);
      // direct: rows chi_i, columns (transition, chi_f)
      tt.clear();
      w.clear();
      wr.clear();
      for (int32_t e : E) {
        tt.get(entries[e].t);
        w.get(entries[e].w_f);
      }
      const size_t nt = tt.back.size();
      std::vector<int32_t> ctab(nt * w.back.size(), -1), cpsi, cwave;
      for (size_t i = 0; i < m; ++i) {
        const dwba_panel_entry_t& x = entries[E[i]];
        ir[i] = wr.get(x.w_i);
        int32_t& c = ctab[(size_t)w.get(x.w_f) * nt + tt.get(x.t)];
        if (c < 0) {
          c = (int32_t)cpsi.size();
          cpsi.push_back(tt.get(x.t));
          cwave.push_back(x.w_f);
        }
        ic[i] = c;
      }
      Panels X, D;
      if (!split_panels(ia, ib, (int)A.u.size(), (int)B.u.size(), E.data(), X)) continue;
      if (!split_panels(ir, ic, (int)wr.back.size(), (int)cpsi.size(), E.data(), D)) continue;
      for (size_t i = 0; i < m; ++i) {
        out->ia[E[i]] = out->n_a + ia[i];
        out->ib[E[i]] = out->n_b + ib[i];
      }
      for (size_t q = 0; q < X.M.size(); ++q) {
        const int g = out->n_exchange++;
        out->x_M[g] = X.M[q];
        out->x_F[g] = X.F[q];
        out->x_set[g] = k;
      }
      for (int32_t v : X.rows) out->x_rows[x_rows++] = out->n_a + v;
      for (int32_t v : X.cols) out->x_cols[x_cols++] = out->n_b + v;
      for (int32_t v : X.entry) out->x_entry[x_ent++] = v;
      for (size_t q = 0; q < D.M.size(); ++q) {
        const int g = out->n_direct++;
        out->d_M[g] = D.M[q];
        out->d_F[g] = D.F[q];
        out->d_set[g] = k;
      }
      for (int32_t v : D.rows) out->d_rows[d_rows++] = wr.back[v];
      for (int32_t v : D.cols) {
        out->d_psi[d_cols] = out->n_psi + cpsi[v];
        out->d_wave[d_cols++] = cwave[v];
      }
      for (int32_t v : D.entry) out->d_entry[d_ent++] = v;
      for (size_t q = 0; q < A.u.size(); ++q) {
        out->a_u[out->n_a] = A.u[q];
        out->a_w[out->n_a] = A.w[q];
        out->a_set[out->n_a++] = k;
      }
      for (size_t q = 0; q < B.u.size(); ++q) {
        out->b_u[out->n_b] = B.u[q];
        out->b_w[out->n_b] = B.w[q];
        out->b_set[out->n_b++] = k;
      }
      for (int32_t t : tt.back) {
        out->psi_t[out->n_psi] = t;
        out->psi_set[out->n_psi++] = k;
      }
    }
  } catch (const std::bad_alloc&) {
    return DWBA_ERR_WORKSPACE;
  }
  return DWBA_OK;
}

extern "C" int dwba_panel_forms(const dwba_panel_t* panels_dev, int n_panels, const dwba_panel_cta_t* ctas_dev,
                                int64_t n_cta, int first_panel, int L_max, double* partial_dev, dwba_stream_t stream) {
  if (n_panels <= 0 || n_cta <= 0) return DWBA_OK;
  if (!panels_dev || !ctas_dev || !partial_dev || first_panel < 0 || L_max < 0 || L_max > DWBA_MAX_L ||
      n_cta > 0x7fffffffLL)
    return DWBA_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  panel_kernel<<<(unsigned)n_cta, P_THREADS, 0, st>>>(panels_dev, ctas_dev, L_max + 1, partial_dev);
  DWBA_CHECK_LAUNCH();
  for (int s0 = 0; s0 < n_panels; s0 += 65535) {
    const int m = n_panels - s0 < 65535 ? n_panels - s0 : 65535;
    const int per = (148 * 8 + m - 1) / m;  // about eight CTAs per SM over all panels
    panel_reduce_kernel<<<dim3(per < 256 ? per : 256, m), 128, 0, st>>>(panels_dev + first_panel + s0, L_max + 1,
                                                                       partial_dev);
    DWBA_CHECK_LAUNCH();
  }
  return DWBA_OK;
}
