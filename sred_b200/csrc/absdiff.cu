// Numerators of the Abs-diff global map: num_p = sum_q |sigma_p - sigma_q| 2^-(a_p - a_q)^2
// (cl/kernelGetGlobalAbsDiffStds2D.cl, kernelGetGlobalAbsDiffStds3D.cl), a = sigma / inv_wscale.
//
// Every term is a function of the two blocks' a alone, so the n sums are one
// function of one variable, with a kink at every a_q. Over the blocks in order of
// a, in slices of 512, the sign of a_p - a_q is constant between slices: the sum over
// the slices below p's minus the sum over those above is smooth in a_p and comes
// from nodes, as the denominators do (weights.cu); only the pairs within a slice
// are evaluated (FP32 terms, FP64 sums of 32).
//   k_abs_keys    a and the index of every block, for the sort (order.cu)
//   k_abs_nodes   one CTA per slice: P[i][s] = sum over slice s of (x_i - a_q) w(x_i, a_q)
//   k_abs_scan    one warp per node: B[i][s] = sum_{s' < s} P[i][s'], A[i][s] = sum_{s' > s} P[i][s'],
//                 each from its far end, so that a small sum is not the difference of larger ones
//   k_abs_eval    one thread per block: B - A interpolated at a_p, plus the slice's pairs
//   k_abs_direct  the blocks that the nodes are not good enough for: all their pairs within
//                 kNodeFar (FP32 terms, FP64 sums)
// A block adds nothing to its own numerator, so one whose nearest neighbours are far, or
// equal, has a sum as small as their weight, while the polynomial's error goes with all that
// is near: 6e-11 of the blocks within a few units, 2e-6 of a sum over blocks 5.5 away, 7e-4
// at 7.5. The 10-point polynomial on the same nodes tells: wherever the 12-point one is off by
// more than 1e-7 the two differ by 2 (blocks 11 away) to 25 times that error (5 away; 12 times
// among equal ones), and where they differ by more than kAbsTol of the numerator, k_abs_direct
// takes the block: an error of 2.5e-6 at most, 4e-7 where terms are not about to vanish; an FP32
// pair term is off by 3e-6.
// n x (nodes + 512) terms instead of n^2 / 2: a map of 500x381, 7x7 (115,000 blocks)
// took 5.6 ms with the pair kernel and takes 0.37. A range of a without a node table (weights.cuh), or one
// whose node-by-slice table exceeds kAbsTable, takes the pair kernel
// (global_fp32.cu), which the device decides (abs_grid).
#include <algorithm>

#include "absdiff.cuh"
#include "epilogue.cuh"

namespace sred {

namespace {

constexpr int kThreads = 256;
constexpr int kPer = kAbsSlice / kThreads;
constexpr int kGroup = 8;  // nodes per step
constexpr double kAbsTol = 5e-6;
constexpr int kFlagWords = kAbsSlice / 32;
constexpr int kParts = 32;  // shares of the slices that a flagged slice's sums are cut into
constexpr int kBlocks = 8;  // flagged blocks at a time

__global__ void k_abs_keys(const BlockParams* __restrict__ params, int n, float* __restrict__ keys,
                           int* __restrict__ idx, int* __restrict__ flagged) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *flagged = 0;
  if (i >= n) return;
  keys[i] = params[i].a;
  idx[i] = i;
}

__global__ void __launch_bounds__(kThreads) k_abs_nodes(const float* __restrict__ keys, const int* __restrict__ order,
                                                        int n, int ns, const unsigned* __restrict__ arange,
                                                        float* __restrict__ sorted, double* __restrict__ table) {
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
    if (i < i1) sorted[i] = v[j];
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

// table: P, replaced by B; above: A.
__global__ void __launch_bounds__(kThreads) k_abs_scan(int ns, const unsigned* __restrict__ arange,
                                                       double* __restrict__ table, double* __restrict__ above) {
  double x0;
  const int m = abs_grid(arange, ns, &x0);
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * kThreads + threadIdx.x) >> 5; i < m; i += gridDim.x * kThreads >> 5) {
    double *row = table + (size_t)i * ns, *up = above + (size_t)i * ns;
    double run = 0.0;
    for (int s0 = (ns - 1) / 32 * 32; s0 >= 0; s0 -= 32) {
      const double p = s0 + lane < ns ? row[s0 + lane] : 0.0;
      double inc = p;
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_down_sync(0xffffffffu, inc, o);
        if (lane + o < 32) inc += t;
      }
      const double next = __shfl_down_sync(0xffffffffu, inc, 1);
      if (s0 + lane < ns) up[s0 + lane] = lane < 31 ? run + next : run;
      run += __shfl_sync(0xffffffffu, inc, 0);
    }
    run = 0.0;
    for (int s0 = 0; s0 < ns; s0 += 32) {
      const double p = s0 + lane < ns ? row[s0 + lane] : 0.0;
      double inc = p;
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      const double before = __shfl_up_sync(0xffffffffu, inc, 1);
      if (s0 + lane < ns) row[s0 + lane] = lane > 0 ? run + before : run;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

// flags: a bit per block of a slice; list: the slices with one, *flagged of them.
__global__ void __launch_bounds__(kThreads) k_abs_eval(const float* __restrict__ sorted, const int* __restrict__ order,
                                                       int n, int ns, const unsigned* __restrict__ arange,
                                                       const double* __restrict__ below,
                                                       const double* __restrict__ above, double inv_wscale,
                                                       double* __restrict__ num, unsigned* __restrict__ flags,
                                                       int* __restrict__ list, int* __restrict__ flagged) {
  double x0;
  if (abs_grid(arange, ns, &x0) == 0) return;
  __shared__ float sa[kAbsSlice];
  const int i0 = blockIdx.x * kAbsSlice, m = min(n - i0, kAbsSlice);
  for (int k = threadIdx.x; k < m; k += kThreads) sa[k] = sorted[i0 + k];
  __syncthreads();
  bool any = false;
#pragma unroll 1
  for (int k = threadIdx.x; k < kAbsSlice; k += kThreads) {
    bool direct = false;
    if (k < m) {
      const float a = sa[k];
      double sum = 0.0;
      for (int q0 = 0; q0 < m; q0 += 32) {
        float part = 0.0f;
        const int q1 = min(m, q0 + 32);
        for (int q = q0; q < q1; q++) {
          const float d = a - sa[q];
          part = fmaf(fabsf(d), ex2_approx(-d * d), part);
        }
        sum += (double)part;
      }
      double est = 0.0;
#pragma unroll
      for (int side = 0; side < 2; side++) {
        double f[12];
        const double s = node_values((double)a, x0, (side ? above : below) + blockIdx.x, ns, f);
        const double v = lagrange<12>(s, f);
        sum += side ? -v : v;
        est += fabs(v - lagrange<10>(s - 1.0, f + 1));
      }
      direct = !(est <= kAbsTol * sum);
      if (!direct) num[order[i0 + k]] = sum * inv_wscale;
    }
    const unsigned bits = __ballot_sync(0xffffffffu, direct);
    if ((threadIdx.x & 31) == 0) flags[blockIdx.x * kFlagWords + (k >> 5)] = bits;
    any |= bits != 0u;
  }
  if (__syncthreads_or(any) && threadIdx.x == 0) list[atomicAdd(flagged, 1)] = blockIdx.x;
}

// A work item: a flagged slice and every kParts-th slice of its pairs' other blocks.
__global__ void __launch_bounds__(kThreads) k_abs_direct(const float* __restrict__ sorted, const int* __restrict__ order,
                                                         int n, int ns, const unsigned* __restrict__ arange,
                                                         double inv_wscale, const unsigned* __restrict__ flags,
                                                         const int* __restrict__ list, const int* __restrict__ flagged,
                                                         double* __restrict__ num) {
  double x0;
  if (abs_grid(arange, ns, &x0) == 0) return;
  __shared__ unsigned bits[kFlagWords];
  __shared__ int at[kAbsSlice];
  __shared__ double red[kThreads / 32][kBlocks];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int item = blockIdx.x; item < *flagged * kParts; item += gridDim.x) {
    const int s = list[item / kParts], part = item % kParts;
    __syncthreads();
    if (threadIdx.x < kFlagWords) bits[threadIdx.x] = flags[s * kFlagWords + threadIdx.x];
    __syncthreads();
    int m = 0;  // the flagged blocks, in order
    for (int j = 0; j < kFlagWords; j++) {
      if ((int)threadIdx.x == j) {
        int o = m;
        for (unsigned b = bits[j]; b; b &= b - 1) at[o++] = s * kAbsSlice + 32 * j + __ffs(b) - 1;
      }
      m += __popc(bits[j]);
    }
    __syncthreads();
    for (int k0 = 0; k0 < m; k0 += kBlocks) {
      float a[kBlocks], some[kBlocks];  // sums of up to 8 terms
      double acc[kBlocks];
      int steps = 0;
#pragma unroll
      for (int k = 0; k < kBlocks; k++) {
        a[k] = sorted[at[min(k0 + k, m - 1)]];
        some[k] = 0.0f;
        acc[k] = 0.0;
      }
      for (int t = part; t < ns; t += kParts) {
        const int i0 = t * kAbsSlice, i1 = min(n, i0 + kAbsSlice);
        if (sorted[i0] > a[kBlocks - 1] + kNodeFar) break;  // (the blocks are in order)
        if (sorted[i1 - 1] < a[0] - kNodeFar) continue;
        float q[kPer];
#pragma unroll
        for (int j = 0; j < kPer; j++) {
          const int i = i0 + j * kThreads + threadIdx.x;
          q[j] = i < i1 ? sorted[i] : 3.4e38f;  // past the end: no weight
        }
#pragma unroll
        for (int k = 0; k < kBlocks; k++) {
#pragma unroll
          for (int j = 0; j < kPer; j++) {
            const float d = a[k] - q[j];
            some[k] = fmaf(fabsf(d), ex2_approx(-d * d), some[k]);
          }
        }
        if ((++steps & 3) == 0) {
#pragma unroll
          for (int k = 0; k < kBlocks; k++) {
            acc[k] += (double)some[k];
            some[k] = 0.0f;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kBlocks; k++) acc[k] += (double)some[k];
      // 8 sums over 32 lanes: lane l ends with sum l & 7
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const bool up = (lane >> r) & 1;
#pragma unroll
        for (int k = 0; k < (kBlocks >> (r + 1)); k++) {
          const double keep = up ? acc[2 * k + 1] : acc[2 * k], send = up ? acc[2 * k] : acc[2 * k + 1];
          acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, 1 << r);
        }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 8);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 16);
      __syncthreads();
      if (lane < kBlocks) red[w][lane] = acc[0];
      __syncthreads();
      if (threadIdx.x < kBlocks && k0 + (int)threadIdx.x < m) {
        double sum = 0.0;
        for (int k = 0; k < kThreads / 32; k++) sum += red[k][threadIdx.x];
        if (sum != 0.0) atomicAdd(num + order[at[k0 + threadIdx.x]], sum * inv_wscale);
      }
    }
  }
}

}  // namespace

int abs_slices(int n) { return (n + kAbsSlice - 1) / kAbsSlice; }

size_t abs_table_doubles(int n) {
  return 2 * std::min<size_t>(kAbsTable, (size_t)kAbsNodes * std::max(1, abs_slices(n)));
}

// (the flags of the slices and their list follow the keys' use: kFlagWords + 1 words a slice, and the count)
size_t abs_keys(int n) { return std::max<size_t>(n, (size_t)(kFlagWords + 1) * abs_slices(n)) + 1; }

cudaError_t launch_absdiff(const BlockParams* params, int n, double inv_wscale, const unsigned* arange, float* keys,
                           int* idx, int* sort_ws, double* table, double* num, int num_sms, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int ns = abs_slices(n);
  int* flagged = reinterpret_cast<int*>(keys + abs_keys(n) - 1);
  k_abs_keys<<<(n + 255) / 256, 256, 0, st>>>(params, n, keys, idx, flagged);
  const int* order;
  const cudaError_t e = launch_sort(keys, idx, n, 0, 3, sort_ws, nullptr, &order, st);
  if (e != cudaSuccess) return e;
  // three passes leave the order in sort_ws: idx holds the sorted keys from here on, and
  // the keys' own array, which k_abs_nodes reads last, the flags and the list of slices
  float* sorted = reinterpret_cast<float*>(idx);
  unsigned* flags = reinterpret_cast<unsigned*>(keys);
  int* list = reinterpret_cast<int*>(flags + (size_t)kFlagWords * ns);
  double* above = table + abs_table_doubles(n) / 2;
  k_abs_nodes<<<ns, kThreads, 0, st>>>(keys, order, n, ns, arange, sorted, table);
  k_abs_scan<<<2 * num_sms, kThreads, 0, st>>>(ns, arange, table, above);
  k_abs_eval<<<ns, kThreads, 0, st>>>(sorted, order, n, ns, arange, table, above, inv_wscale, num, flags, list,
                                      flagged);
  k_abs_direct<<<4 * num_sms, kThreads, 0, st>>>(sorted, order, n, ns, arange, inv_wscale, flags, list, flagged, num);
  return cudaGetLastError();
}

}  // namespace sred
