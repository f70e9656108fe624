// Ordering of the compacted blocks by standard deviation (order.cu).
#pragma once
#include "common.cuh"

namespace sred {

constexpr int kSortSpan = 4096;  // blocks per CTA of a pass

// Ints of workspace launch_sort_blocks needs for n blocks.
size_t sort_workspace_ints(int n);

// Sorts pix[0, n) (pixel indices) by stds[pix] in place, ties in list order,
// and rewrites slot[pix[j]] = j.
cudaError_t launch_sort_blocks(const float* stds, int* pix, int n, int* ws, int* slot, cudaStream_t st);
constexpr int kSortLaunches = 6;

}  // namespace sred
