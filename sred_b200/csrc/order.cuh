// Stable radix sort of an index list by float keys (order.cu).
#pragma once
#include "common.cuh"

namespace sred {

constexpr int kSortSpan = 2048;  // list entries per CTA of a pass

// Ints of workspace launch_sort needs for n entries.
size_t sort_workspace_ints(int n);

// Sorts idx[0, n) by bits [shift, shift + 11 passes) of keys[idx] (the sign
// dropped; passes <= 3), ties in list order. *sorted: the sorted list (idx itself
// after two passes, part of ws after an odd number). slot (nullable): the sort
// writes slot[entry] = its position.
cudaError_t launch_sort(const float* keys, int* idx, int n, int shift, int passes, int* ws, int* slot,
                        const int** sorted, cudaStream_t st);
constexpr int kStdShift = 9, kStdPasses = 2;  // blocks by std (launch count: 3 a pass)

}  // namespace sred
