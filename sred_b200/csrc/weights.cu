// Denominators of the global maps: den_p = sum_q 2^-(a_p - a_q)^2 over the
// contracted blocks (the weight's own sum, java/CLUtils.java:1747-1770), the
// self pair included.
//
// The weight depends on the two blocks' scalars a alone, so the n sums are one
// function of one variable, F(x) = sum_q 2^-(x - a_q)^2, at the points a_p. F is
// a sum of Gaussians of one width: between nodes 1/8 apart a 12-point Lagrange
// polynomial reproduces it to 6e-11 of the number of blocks near x (the 12th derivative
// of 2^-x^2 is at most 7.4e4; times 5.5e-5 h^12). The self pair keeps every sum above 1;
// a block 4.25 units away from a million others has a sum near 5 and an error of 3e-8 of
// it. So the sums take n terms at some tens of
// nodes (FP64) and n interpolations instead of n^2 / 2 pair terms; accumulating
// them beside the numerators was a sixth of the pair arithmetic and half of the
// contraction's accumulators.
//
// k_den_nodes: one CTA per 2,048 blocks, eight nodes at a time; consecutive
// nodes of a block follow from two multiplications,
//   2^-(x + h - a)^2 = 2^-(x - a)^2 * r,  r = 2^-(2 (x - a) h + h^2),  r' = r 2^(-2 h^2),
// and one FP64 atomic add per node and CTA. Nodes further than 14 from every
// block of the slice (terms below 2^-169) are skipped. Few slices share their nodes
// out among several CTAs each: 6.5 us instead of 26 for 9,810 blocks.
// A slice of a wide range steps over the groups of nodes that none of its blocks is near.
// k_den_eval: one thread per block. Where the range of a does not fit the node
// table (32,766 at h = 1/8) or is not finite, the same kernel sums the pair terms
// directly (FP32 terms, FP64 sums of 256), slice by slice within that distance. A range of
// 4,500 (256x256, 5x5 Pearson, a nearly silent background; the table once ended at 2,046)
// takes 1.17 ms by nodes, 1.93 directly.
#include <algorithm>

#include "epilogue.cuh"
#include "weights.cuh"

namespace sred {

namespace {

constexpr int kThreads = 256;
constexpr int kPer = kDenSlice / kThreads;
constexpr int kGroup = 8;          // nodes per step
constexpr int kDenCtas = 4 * 148;  // CTAs that few slices are spread over

__global__ void __launch_bounds__(kThreads) k_den_nodes(const BlockParams* __restrict__ params, int n,
                                                        const unsigned* __restrict__ arange,
                                                        double* __restrict__ nodes, float2* __restrict__ slices) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i0 = blockIdx.x * kDenSlice;
  __shared__ float2 wr[kThreads / 32];
  __shared__ double red[kThreads / 32][kGroup];
  float v[kPer];
  float lo = 3.4e38f, hi = -3.4e38f;
  bool bad = false;
#pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = i0 + j * kThreads + threadIdx.x;
    v[j] = i < n ? params[i].a : 3.4e38f;  // past the end: further than kNodeFar from every node
    if (i < n) {
      lo = fminf(lo, v[j]);
      hi = fmaxf(hi, v[j]);
      bad |= !(v[j] - v[j] == 0.0f);
    }
  }
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (__any_sync(0xffffffffu, bad)) lo = hi = nanf("");
  if (lane == 0) wr[w] = make_float2(lo, hi);
  __syncthreads();
  lo = wr[0].x;
  hi = wr[0].y;
  bad = lo != lo;
  for (int k = 1; k < kThreads / 32; k++) {
    bad |= wr[k].x != wr[k].x;
    lo = fminf(lo, wr[k].x);
    hi = fmaxf(hi, wr[k].y);
  }
  if (bad) lo = hi = nanf("");
  if (threadIdx.x == 0 && blockIdx.y == 0) slices[blockIdx.x] = make_float2(lo, hi);
  double x0;
  const int m = node_grid(arange, &x0);
  if (m == 0) return;
  const int g0 = max(0, (int)floor(((double)lo - kNodeFar - x0) / (kNodeH * kGroup)));
  const int g1 = min((m - 1) / kGroup, (int)floor(((double)hi + kNodeFar - x0) / (kNodeH * kGroup)));
  const double q = exp2(-2.0 * kNodeH * kNodeH);
  for (int g = g0 + blockIdx.y; g <= g1; g += gridDim.y) {
    const double xb = x0 + (double)(g * kGroup) * kNodeH;
    if (g1 - g0 > 64) {
      const float xc = (float)(xb + 0.5 * kNodeH * kGroup);
      bool near = false;
#pragma unroll
      for (int j = 0; j < kPer; j++) near |= fabsf(xc - v[j]) <= kNodeFar + 0.5f;
      if (!__syncthreads_or(near)) continue;
    }
    double acc[kGroup];
#pragma unroll
    for (int k = 0; k < kGroup; k++) acc[k] = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const double d = xb - (double)v[j];
      if (fabs(d + 0.5 * kNodeH * kGroup) > (double)kNodeFar) continue;  // (2^-182 at most)
      double e = exp2(-d * d), r = exp2(-(2.0 * d + kNodeH) * kNodeH);
#pragma unroll
      for (int k = 0; k < kGroup; k++) {
        acc[k] += e;
        e *= r;
        r *= q;
      }
    }
    // 8 sums over 32 lanes: three halving steps leave lane l sum index l & 7, two more finish it
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
      atomicAdd(nodes + g * kGroup + threadIdx.x, t);
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_den_eval(const BlockParams* __restrict__ params, int n,
                                                       const unsigned* __restrict__ arange,
                                                       const double* __restrict__ nodes,
                                                       const float2* __restrict__ slices, int nslices,
                                                       double* __restrict__ den) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  double x0;
  if (node_grid(arange, &x0) > 0) {
    if (i >= n) return;
    den[i] = interpolate12((double)params[i].a, x0, nodes, 1);
    return;
  }
  __shared__ float sa[kThreads];
  __shared__ float2 wr[kThreads / 32];
  const float a = i < n ? params[i].a : 0.0f;
  float lo = i < n ? a : 3.4e38f, hi = i < n ? a : -3.4e38f;
  const bool bad = i < n && !(a - a == 0.0f);
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const bool any_bad = __syncthreads_or(bad);
  if ((threadIdx.x & 31) == 0) wr[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  for (int k = 0; k < kThreads / 32; k++) {
    lo = fminf(lo, wr[k].x);
    hi = fmaxf(hi, wr[k].y);
  }
  double sum = 0.0;
  for (int s = 0; s < nslices; s++) {
    const float2 r = slices[s];
    if (!any_bad && (r.x - hi > kNodeFar || lo - r.y > kNodeFar)) continue;  // (a NaN range is not skipped)
    const int q0 = s * kDenSlice, q1 = min(n, q0 + kDenSlice);
    for (int qb = q0; qb < q1; qb += kThreads) {
      const int m = min(kThreads, q1 - qb);
      __syncthreads();
      if ((int)threadIdx.x < m) sa[threadIdx.x] = params[qb + threadIdx.x].a;
      __syncthreads();
      float part = 0.0f;
      for (int k = 0; k < m; k++) {
        const float d = a - sa[k];
        part += ex2_approx(-d * d);
      }
      sum += (double)part;
    }
  }
  if (i < n) den[i] = sum;
}

}  // namespace

int den_slices(int n) { return (n + kDenSlice - 1) / kDenSlice; }

cudaError_t launch_den(const BlockParams* params, int n, const unsigned* arange, double* nodes, float2* slices,
                       double* den, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(nodes, 0, kDenNodes * sizeof(double), st);
  if (e != cudaSuccess) return e;
  const int ns = den_slices(n);
  const int parts = std::max(1, std::min(32, kDenCtas / ns));
  k_den_nodes<<<dim3(ns, parts), kThreads, 0, st>>>(params, n, arange, nodes, slices);
  k_den_eval<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(params, n, arange, nodes, slices, ns, den);
  return cudaGetLastError();
}

}  // namespace sred
