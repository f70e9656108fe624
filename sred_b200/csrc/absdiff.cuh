// Numerators of the Abs-diff global map from the blocks' weight arguments (absdiff.cu).
#pragma once
#include "order.cuh"
#include "weights.cuh"

namespace sred {

constexpr int kAbsSlice = 512;         // blocks per slice, in order of a
constexpr int kAbsTable = 4 << 20;     // doubles of one node-by-slice table, at most
constexpr int kAbsNodes = 1 << 16;     // nodes of the tables, at most

// Nodes of the tables for ns slices and its first node (0: the pair kernel runs instead).
__device__ __forceinline__ int abs_grid(const unsigned* __restrict__ arange, int ns, double* x0) {
  const int m = node_grid(arange, x0);
  return m <= kAbsNodes && (long long)m * ns <= kAbsTable ? m : 0;
}

int abs_slices(int n);
// Doubles of workspace for the two node-by-slice tables, and keys (or indices) for n blocks.
size_t abs_table_doubles(int n);
size_t abs_keys(int n);

// num[p] for the n blocks of params (zeroed by the caller), where abs_grid gives a
// table; otherwise num is left as it is. arange: as for launch_den; keys and idx:
// abs_keys(n) entries each, sort_ws: sort_workspace_ints(n) ints, table:
// abs_table_doubles(n) doubles of workspace.
cudaError_t launch_absdiff(const BlockParams* params, int n, double inv_wscale, const unsigned* arange, float* keys,
                           int* idx, int* sort_ws, double* table, double* num, int num_sms, cudaStream_t st);
constexpr int kAbsLaunches = 5 + 9;

}  // namespace sred
