// 3D (volume) block repetition maps: device kernels and host helpers.
#pragma once
#include "common.cuh"

namespace sred {

constexpr int kMaxK3 = 4096;  // largest ellipsoid block size accepted

// A W x H x D volume ([D][H][W] floats) and the ellipsoid block radii; k is
// the number of voxels of the ellipsoid.
struct Vol3 {
  int W, H, D;
  int rw, rh, rd;
  int k;
  int z0 = 0;  // first slice of a launch over slices [z0, z0 + gridDim.z) of the per-voxel kernels
  int nrows = 0;  // rows of the ellipsoid
};

// Host: linear offsets (z W H + y W + x) of the voxels of the ellipsoid
// inscribed in a bw x bh x bd block, z-y-x order (java/Utils.java:1075-1085,
// float arithmetic). Writes at most kMaxK3 offsets; returns the voxel count.
int build_ellipsoid(int bw, int bh, int bd, int W, int H, int* off);

// One thread per voxel; dynamic shared memory: k ints.
__global__ void k_local_stats3d(const float* img, Vol3 v, const int* off, float* means, float* stds);
// The 3D block map over slices [v.z0, z1), NRMSE inverted and Abs-diff turned into
// 1 - x; the local stds (stds, or null) and the range of the interior (mm, or null).
// off: the block's offsets and rows (prepare_volume).
cudaError_t launch_block_map3d(const float* img, Vol3 v, const int* off, const float* ref, float ref_mean,
                               float ref_std, int metric, float* out, float* stds, unsigned* mm, cudaStream_t st,
                               int z1);
__global__ void k_divide_fixed(const float* a, size_t n, float b, float* out);
__global__ void k_divide_fixed64(const double* a, size_t n, double b, double* out);
// The FP32 sum of sigma^2 over the interior in raster order (0 without an interior).
cudaError_t launch_noise3d(const float* stds, Vol3 v, float* sum, cudaStream_t st);
__global__ void k_mask3d(const float* stds, Vol3 v, float thr, float* mask, float* map);

// 3D global map (the 2D pair engines run on the compacted block lists).
__global__ void k_flags3d(const float* stds, Vol3 v, float thr, int flat_columns, float* mask, uint8_t* flags,
                          unsigned long long* n_mask);
__global__ void k_finalize3d(const int* slot, Vol3 v, const double* num, const double* den,
                             const BlockParams* params, int n_flat, int metric, double sk, double n_pixels,
                             const float* mask, int apply_mask, float* out);

}  // namespace sred
