// Denominators of the global maps from the blocks' weight arguments (weights.cu).
#pragma once
#include "common.cuh"

namespace sred {

constexpr int kDenSlice = 2048;    // blocks per CTA of the node sums
constexpr int kDenNodes = 1 << 18; // node table (doubles): a-ranges of up to 32,766

// Functions of a block's a as sums over all blocks: nodes kNodeH apart and a
// 12-point Lagrange polynomial between them (weights.cu: how accurate).
constexpr double kNodeH = 0.125;
constexpr int kNodePad = 6;        // nodes below the smallest a
constexpr float kNodeFar = 14.0f;  // terms further off (2^-169) are left out

// Node grid of the a-range (arange: see launch_den): first node and count (0: no grid).
__device__ __forceinline__ int node_grid(const unsigned* __restrict__ arange, double* x0) {
  const unsigned lo = ~arange[0], hi = arange[1];
  if (hi >= 0x7f800000u) return 0;  // infinite or NaN (either sign)
  const double a0 = (double)__uint_as_float(lo), a1 = (double)__uint_as_float(hi);
  *x0 = a0 - kNodePad * kNodeH;
  const double m = floor((a1 - a0) / kNodeH) + 2 * kNodePad + 2;
  return m <= (double)kDenNodes ? (int)m : 0;
}

// 1 / prod_{j != k} (k - j) for the nodes 0..N-1 (N even).
template <int N>
__device__ __forceinline__ double lagrange_scale(int k) {
  const double f[12] = {1.0, 1.0, 2.0, 6.0, 24.0, 120.0, 720.0, 5040.0, 40320.0, 362880.0, 3628800.0, 39916800.0};
  const double v = 1.0 / (f[k] * f[N - 1 - k]);
  return (k & 1) ? v : -v;  // sign (-1)^(N - 1 - k)
}

// The polynomial through the values f[0..N-1] at the nodes 0..N-1, at s.
template <int N>
__device__ __forceinline__ double lagrange(double s, const double* f) {
  double suf[N];
  suf[N - 1] = 1.0;
#pragma unroll
  for (int k = N - 1; k > 0; k--) suf[k - 1] = suf[k] * (s - (double)k);
  double pre = 1.0, sum = 0.0;
#pragma unroll
  for (int k = 0; k < N; k++) {
    sum += lagrange_scale<N>(k) * pre * suf[k] * f[k];
    pre *= s - (double)k;
  }
  return sum;
}

// The 12 node values around a (stride between nodes), and a's place among them (in [5, 6)).
__device__ __forceinline__ double node_values(double a, double x0, const double* __restrict__ nodes, size_t stride,
                                              double (&f)[12]) {
  const double t = (a - x0) / kNodeH;
  const int k0 = (int)floor(t) - (kNodePad - 1);
#pragma unroll
  for (int k = 0; k < 12; k++) f[k] = nodes[(size_t)(k0 + k) * stride];
  return t - (double)k0;
}

// The function at a from its node values.
__device__ __forceinline__ double interpolate12(double a, double x0, const double* __restrict__ nodes, size_t stride) {
  double f[12];
  const double s = node_values(a, x0, nodes, stride, f);
  return lagrange<12>(s, f);
}

int den_slices(int n);

// den[p] = sum_q 2^-(a_p - a_q)^2 over the n blocks of params. arange: the
// complemented bits of the smallest a and the bits of the largest one (both
// maxima over unsigned words, from 0; a >= 0, and a NaN or infinity shows in the
// second); nodes: kDenNodes doubles and slices: den_slices(n) pairs of workspace.
cudaError_t launch_den(const BlockParams* params, int n, const unsigned* arange, double* nodes, float2* slices,
                       double* den, cudaStream_t st);
constexpr int kDenLaunches = 2;

}  // namespace sred
