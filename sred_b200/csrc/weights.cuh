// Denominators of the global maps from the blocks' weight arguments (weights.cu).
#pragma once
#include "common.cuh"

namespace sred {

constexpr int kDenSlice = 2048;    // blocks per CTA of the node sums
constexpr int kDenNodes = 16384;   // node table (doubles)

int den_slices(int n);

// den[p] = sum_q 2^-(a_p - a_q)^2 over the n blocks of params. arange: the
// complemented bits of the smallest a and the bits of the largest one (both
// maxima over unsigned words, from 0; a >= 0, and a NaN or infinity shows in the
// second); nodes: kDenNodes doubles and slices: den_slices(n) pairs of workspace.
cudaError_t launch_den(const BlockParams* params, int n, const unsigned* arange, double* nodes, float2* slices,
                       double* den, cudaStream_t st);
constexpr int kDenLaunches = 2;

}  // namespace sred
