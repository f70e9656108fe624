// Ordering of the relevant blocks: a stable radix sort of an index list by
// non-negative float keys, 11 bits a pass, ties in list order. Deterministic:
// ranks come from counts in list order, never from the order in which atomics land.
//   - the tensor-core engine's weights (global_tc.cu): the compacted pixel list by
//     the top 22 bits below the sign of the FP32 local std (8 exponent and 14
//     mantissa bits, so neighbours differ by less than 2^-14 relative beyond a true
//     order), two passes;
//   - Abs-diff (absdiff.cu): the blocks by all 31 bits of a, three passes.
//
// Bound by latency (a few CTAs' worth of work and three launches a pass).
#include "order.cuh"

#include <utility>

namespace sred {

namespace {

constexpr int kDigitBits = 11;
constexpr int kBins = 1 << kDigitBits;
constexpr int kWarps = 8, kThreads = 32 * kWarps;
constexpr int kPerWarp = kSortSpan / kWarps;
constexpr int kScanBins = 32;  // bins per CTA of the scan

// Digit of a key: the float bits without the sign (a NaN sorts last).
__device__ __forceinline__ unsigned sort_digit(float s, int shift) {
  return ((__float_as_uint(s) & 0x7fffffffu) >> shift) & (kBins - 1);
}

// table[bin][span]: blocks of each span with that digit; total[bin]: of all spans.
__global__ void __launch_bounds__(kThreads) k_sort_count(const float* __restrict__ keys, const int* __restrict__ idx,
                                                         int n, int shift, int nspan, int* __restrict__ table,
                                                         int* __restrict__ total) {
  __shared__ int h[kBins];
  for (int i = threadIdx.x; i < kBins; i += kThreads) h[i] = 0;
  __syncthreads();
  const int i0 = blockIdx.x * kSortSpan, i1 = min(n, i0 + kSortSpan);
  for (int i = i0 + threadIdx.x; i < i1; i += kThreads) atomicAdd(h + sort_digit(keys[idx[i]], shift), 1);
  __syncthreads();
  for (int b = threadIdx.x; b < kBins; b += kThreads) {
    const int c = h[b];
    table[(size_t)b * nspan + blockIdx.x] = c;
    if (c) atomicAdd(total + b, c);
  }
}

// table[bin][span] -> first output position of that bin's blocks of that span.
// One CTA per 32 bins, one warp per bin.
__global__ void __launch_bounds__(kThreads) k_sort_scan(const int* __restrict__ total, int nspan,
                                                        int* __restrict__ table) {
  __shared__ int part[kWarps], first[kScanBins];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b0 = blockIdx.x * kScanBins;
  int s = 0;
  for (int i = threadIdx.x; i < b0; i += kThreads) s += total[i];
  s = __reduce_add_sync(0xffffffffu, s);
  if (lane == 0) part[w] = s;
  __syncthreads();
  if (w == 0) {
    int base = 0;
    for (int i = 0; i < kWarps; i++) base += part[i];
    const int t = total[b0 + lane];
    int inc = t;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    first[lane] = base + inc - t;
  }
  __syncthreads();
  for (int k = w; k < kScanBins; k += kWarps) {
    int* row = table + (size_t)(b0 + k) * nspan;
    int run = first[k];
    for (int j0 = 0; j0 < nspan; j0 += 32) {
      const int t = j0 + lane < nspan ? row[j0 + lane] : 0;
      int inc = t;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (j0 + lane < nspan) row[j0 + lane] = run + inc - t;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

// Stable scatter of one span: every warp takes its part of the span in order;
// blocks of equal digit in a warp's step are ranked by lane (match_any).
__global__ void __launch_bounds__(kThreads) k_sort_scatter(const float* __restrict__ keys, const int* __restrict__ idx,
                                                           int n, int shift, int nspan, const int* __restrict__ table,
                                                           int* __restrict__ out, int* __restrict__ slot) {
  extern __shared__ int cnt[];  // [kWarps][kBins]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kWarps * kBins; i += kThreads) cnt[i] = 0;
  __syncthreads();
  int* mine = cnt + w * kBins;
  const int i0 = blockIdx.x * kSortSpan + w * kPerWarp;
  int px[kPerWarp / 32], dg[kPerWarp / 32];
#pragma unroll
  for (int j = 0; j < kPerWarp / 32; j++) {
    const int i = i0 + 32 * j + lane;
    px[j] = i < n ? idx[i] : -1;
    dg[j] = px[j] >= 0 ? (int)sort_digit(keys[px[j]], shift) : -1;
    if (dg[j] >= 0) atomicAdd(mine + dg[j], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kBins; b += kThreads) {
    int run = table[(size_t)b * nspan + blockIdx.x];
    for (int v = 0; v < kWarps; v++) {
      const int c = cnt[v * kBins + b];
      cnt[v * kBins + b] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPerWarp / 32; j++) {
    const unsigned peers = __match_any_sync(0xffffffffu, dg[j]);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int base = 0;
    if (dg[j] >= 0) base = mine[dg[j]];
    __syncwarp();
    if (dg[j] >= 0) {
      if (rank == 0) mine[dg[j]] = base + __popc(peers);
      const int o = base + rank;
      out[o] = px[j];
      if (slot) slot[px[j]] = o;
    }
    __syncwarp();
  }
}

}  // namespace

size_t sort_workspace_ints(int n) {
  const size_t nspan = ((size_t)n + kSortSpan - 1) / kSortSpan;
  return (size_t)kBins * nspan + 3 * kBins + (size_t)n;
}

cudaError_t launch_sort(const float* keys, int* idx, int n, int shift, int passes, int* ws, int* slot,
                        const int** sorted, cudaStream_t st) {
  if (sorted) *sorted = idx;
  if (n <= 0) return cudaSuccess;
  const int nspan = (n + kSortSpan - 1) / kSortSpan;
  int* total = ws;                           // [passes][kBins]
  int* table = total + 3 * kBins;            // [kBins][nspan]
  int* tmp = table + (size_t)kBins * nspan;  // [n]
  const int smem = kWarps * kBins * (int)sizeof(int);
  cudaError_t e = cudaFuncSetAttribute(k_sort_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(total, 0, passes * kBins * sizeof(int), st);
  if (e != cudaSuccess) return e;
  int *in = idx, *out = tmp;
  for (int pass = 0; pass < passes; pass++) {
    const int sh = shift + kDigitBits * pass;
    k_sort_count<<<nspan, kThreads, 0, st>>>(keys, in, n, sh, nspan, table, total + pass * kBins);
    k_sort_scan<<<kBins / kScanBins, kThreads, 0, st>>>(total + pass * kBins, nspan, table);
    k_sort_scatter<<<nspan, kThreads, smem, st>>>(keys, in, n, sh, nspan, table, out,
                                                  pass + 1 == passes ? slot : nullptr);
    std::swap(in, out);
  }
  if (sorted) *sorted = in;
  return cudaGetLastError();
}

}  // namespace sred
