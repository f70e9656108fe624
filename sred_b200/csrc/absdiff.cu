// Numerators of the Abs-diff global map: num_p = sum_q |sigma_p - sigma_q| 2^-(a_p - a_q)^2
// (cl/kernelGetGlobalAbsDiffStds2D.cl, kernelGetGlobalAbsDiffStds3D.cl), a = sigma / inv_wscale.
//
// Every term is a function of the two blocks' a alone, so the n sums are one
// function of one variable, with a kink at every a_q. Over the blocks in order of
// a, in slices of 512, the sign of a_p - a_q is constant between slices: the sum over
// the slices below p's minus the sum over those above is smooth in a_p and comes
// from nodes, as the denominators do (weights.cu); only the pairs within a slice
// are evaluated (FP32 terms, FP64 sums of 32).
//   k_abs_keys   a and the index of every block, for the sort (order.cu)
//   k_abs_nodes  one CTA per slice: P[i][s] = sum over slice s of (x_i - a_q) w(x_i, a_q)
//   k_abs_scan   one warp per node: T[i][s] = sum_{s' < s} P[i][s'] - sum_{s' > s} P[i][s']
//   k_abs_eval   one thread per block: T interpolated at a_p, plus the slice's pairs
// n x (nodes + 512) terms instead of n^2 / 2: a map of 500x381, 7x7 (115,000 blocks)
// took 5.6 ms with the pair kernel and takes 0.48. A range of a without a node table (weights.cuh), or one
// whose node-by-slice table exceeds kAbsTable, takes the pair kernel
// (global_fp32.cu), which the device decides (abs_grid).
#include "absdiff.cuh"
#include "epilogue.cuh"

namespace sred {

namespace {

constexpr int kThreads = 256;
constexpr int kPer = kAbsSlice / kThreads;
constexpr int kGroup = 8;  // nodes per step

__global__ void k_abs_keys(const BlockParams* __restrict__ params, int n, float* __restrict__ keys,
                           int* __restrict__ idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = params[i].a;
  idx[i] = i;
}

__global__ void __launch_bounds__(kThreads) k_abs_nodes(const float* __restrict__ keys, const int* __restrict__ order,
                                                        int n, int ns, const unsigned* __restrict__ arange,
                                                        double* __restrict__ table) {
  double x0;
  const int m = abs_grid(arange, ns, &x0);
  if (m == 0) return;
  __shared__ double red[kThreads / 32][kGroup];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = blockIdx.x * kAbsSlice, i1 = min(n, i0 + kAbsSlice);
  const float lo = keys[order[i0]], hi = keys[order[i1 - 1]];
  float v[kPer];
#pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = i0 + j * kThreads + threadIdx.x;
    v[j] = i < i1 ? keys[order[i]] : 3.4e38f;  // past the end: further than kNodeFar from every node
  }
  const double q = exp2(-2.0 * kNodeH * kNodeH);
  for (int g = 0; g * kGroup < m; g++) {
    const double xb = x0 + (double)(g * kGroup) * kNodeH;
    if (xb + kGroup * kNodeH < (double)lo - kNodeFar || xb > (double)hi + kNodeFar) {
      if (threadIdx.x < kGroup && g * kGroup + (int)threadIdx.x < m)
        table[(size_t)(g * kGroup + threadIdx.x) * ns + blockIdx.x] = 0.0;
      continue;
    }
    double acc[kGroup];
#pragma unroll
    for (int k = 0; k < kGroup; k++) acc[k] = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const double d = xb - (double)v[j];
      if (fabs(d + 0.5 * kNodeH * kGroup) > (double)kNodeFar) continue;
      double e = exp2(-d * d), r = exp2(-(2.0 * d + kNodeH) * kNodeH), t = d;
#pragma unroll
      for (int k = 0; k < kGroup; k++) {
        acc[k] += t * e;
        e *= r;
        r *= q;
        t += kNodeH;
      }
    }
    // 8 sums over 32 lanes: lane l ends with sum l & 7
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const bool up = (lane >> s) & 1;
#pragma unroll
      for (int k = 0; k < (kGroup >> (s + 1)); k++) {
        const double keep = up ? acc[2 * k + 1] : acc[2 * k], send = up ? acc[2 * k] : acc[2 * k + 1];
        acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, 1 << s);
      }
    }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 8);
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 16);
    __syncthreads();
    if (lane < kGroup) red[w][lane] = acc[0];
    __syncthreads();
    if (threadIdx.x < kGroup && g * kGroup + (int)threadIdx.x < m) {
      double t = 0.0;
      for (int k = 0; k < kThreads / 32; k++) t += red[k][threadIdx.x];
      table[(size_t)(g * kGroup + threadIdx.x) * ns + blockIdx.x] = t;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_abs_scan(int ns, const unsigned* __restrict__ arange,
                                                       double* __restrict__ table) {
  double x0;
  const int m = abs_grid(arange, ns, &x0);
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * kThreads + threadIdx.x) >> 5; i < m; i += gridDim.x * kThreads >> 5) {
    double* row = table + (size_t)i * ns;
    double total = 0.0;
    for (int s = lane; s < ns; s += 32) total += row[s];
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    double below = 0.0;
    for (int s0 = 0; s0 < ns; s0 += 32) {
      const double p = s0 + lane < ns ? row[s0 + lane] : 0.0;
      double inc = p;
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      const double before = below + (inc - p);
      if (s0 + lane < ns) row[s0 + lane] = 2.0 * before + p - total;  // before - (total - before - p)
      below += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_abs_eval(const float* __restrict__ keys, const int* __restrict__ order,
                                                       int n, int ns, const unsigned* __restrict__ arange,
                                                       const double* __restrict__ table, double inv_wscale,
                                                       double* __restrict__ num) {
  double x0;
  if (abs_grid(arange, ns, &x0) == 0) return;
  __shared__ float sa[kAbsSlice];
  const int i0 = blockIdx.x * kAbsSlice, m = min(n - i0, kAbsSlice);
  for (int k = threadIdx.x; k < m; k += kThreads) sa[k] = keys[order[i0 + k]];
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += kThreads) {
    const float a = sa[k];
    double near = 0.0;
    for (int q0 = 0; q0 < m; q0 += 32) {
      float part = 0.0f;
      const int q1 = min(m, q0 + 32);
      for (int q = q0; q < q1; q++) {
        const float d = a - sa[q];
        part = fmaf(fabsf(d), ex2_approx(-d * d), part);
      }
      near += (double)part;
    }
    num[order[i0 + k]] = (interpolate12((double)a, x0, table + blockIdx.x, ns) + near) * inv_wscale;
  }
}

}  // namespace

int abs_slices(int n) { return (n + kAbsSlice - 1) / kAbsSlice; }

cudaError_t launch_absdiff(const BlockParams* params, int n, double inv_wscale, const unsigned* arange, float* keys,
                           int* idx, int* sort_ws, double* table, double* num, int num_sms, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int ns = abs_slices(n);
  k_abs_keys<<<(n + 255) / 256, 256, 0, st>>>(params, n, keys, idx);
  const int* order;
  const cudaError_t e = launch_sort(keys, idx, n, 0, 3, sort_ws, nullptr, &order, st);
  if (e != cudaSuccess) return e;
  k_abs_nodes<<<ns, kThreads, 0, st>>>(keys, order, n, ns, arange, table);
  k_abs_scan<<<2 * num_sms, kThreads, 0, st>>>(ns, arange, table);
  k_abs_eval<<<ns, kThreads, 0, st>>>(keys, order, n, ns, arange, table, inv_wscale, num);
  return cudaGetLastError();
}

}  // namespace sred
