// Phase-interval helpers shared by the node-set kernels (nodes.cu, cupy_nodes.cu): the breakpoints
// of generate_phase_nodes (oscillatory_integrals.py:1625-1713) -- numpy.linspace arithmetic when no
// breakpoint list is given -- and the search for the interval containing a radius.
#pragma once
#include "common.cuh"

namespace dwba_nodes {

constexpr int MAX_CC = 15;

struct SetView {
  const double* r;
  const double* lr;
  const double* br;  // breakpoints or nullptr (linspace)
  int n_grid, n1, n_int, log1, log2;
  double start, stop, step;
  double inv_step;  // 1/step, for the search of an interval
};

__device__ __forceinline__ void interval(const SetView& s, int m, double& a, double& b) {
  if (s.br != nullptr) {
    a = s.br[m];
    b = s.br[m + 1];
  } else {  // numpy.linspace: y[i] = i*step + start, y[num-1] = stop
    a = rn_add(rn_mul((double)m, s.step), s.start);
    b = (m + 1 == s.n_int) ? s.stop : rn_add(rn_mul((double)(m + 1), s.step), s.start);
  }
}

// left end of interval m (right end of interval m - 1, except that the last one ends at `stop`)
__device__ __forceinline__ double interval_start(const SetView& s, int m) {
  return s.br != nullptr ? s.br[m] : rn_add(rn_mul((double)m, s.step), s.start);
}
__device__ __forceinline__ double interval_end(const SetView& s, int m) {
  return (s.br == nullptr && m + 1 == s.n_int) ? s.stop : interval_start(s, m + 1);
}

// last interval m whose left end a_m <= x (0 if none)
__device__ __forceinline__ int interval_floor(const SetView& s, double x) {
  if (s.br != nullptr) {
    int lo = 0, hi = s.n_int;  // a_lo <= x < a_hi
    if (!(s.br[0] <= x)) return 0;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s.br[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
  }
  double q = floor((x - s.start) * s.inv_step);
  int m = q < 0.0 ? 0 : (q > (double)(s.n_int - 1) ? s.n_int - 1 : (int)q);
  // the closed form can be off after rounding: correct against the exact left ends
  while (m > 0 && interval_start(s, m) > x) --m;
  while (m + 1 < s.n_int && interval_start(s, m + 1) <= x) ++m;
  return m;
}

}  // namespace dwba_nodes
