// Kernel declarations shared between the device translation units and the
// host orchestration (sred_api.cu).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace sred {

constexpr int kCompactSeg = 2048;

struct RefBlock {
  int k;
  float mean, std;
  float px[kMaxK];
};

// moments.cu
__global__ void k_local_stats(const float* img, int W, int H, Ellipse e, float* means, float* stds);
__global__ void k_noise_tiles(const float* img, int W, int t, int nbx, int nb, float* vars, int* bad);
__global__ void k_flags(const float* stds, const float* mask_in, int W, int H, int rw, int rh, float thr,
                        float* mask, uint8_t* flags, unsigned long long* n_mask);
__global__ void k_count(const uint8_t* flags, size_t n, int2* counts);
__global__ void k_scan(int2* counts, int nseg);
__global__ void k_scatter(const uint8_t* flags, size_t n, const int2* offs, int* gram_pix, int* flat_pix,
                          int* slot);
// The listed blocks' parameters and operands; off: the block's linear offsets (3D), or
// null for e on an image W wide.
cudaError_t launch_pack(const float* img, int W, const Ellipse& e, const int* off, int K, const int* gram_pix, int n,
                        float wscale, float* U, int kp, __half* S, BlockParams* params, float* tile_rmax, double* sums,
                        unsigned* arange, int num_sms, cudaStream_t st);
__global__ void k_finalize(const int* slot, int W, int H, int rw, int rh, const double* num, const double* den,
                           const BlockParams* params, const double* sums, int n_flat, int metric, double sk,
                           double n_pixels, const float* mask, int apply_mask, float* out);
__global__ void k_pack_vectors(const float* u, int n, int K, float scale, float* U, int kp, __half* S);
// Per-plane min/max words before a range is taken: {ordered +inf, ordered -inf} per plane
// (a kernel rather than a copy from pageable host memory, which would wait
// for the stream to drain).
__global__ void k_init_minmax(unsigned* mm, int planes);

// block_map.cu
// The map of a reference block (all metrics of block_metric_value), the local stds
// (stds, or null) and the range of the interior (mm, or null: 2 words per frame).
cudaError_t launch_block_map(const float* img, int w, int h, int frames, const Ellipse& e, const RefBlock& rb,
                             int metric, float* out, float* stds, unsigned* mm, int num_sms, cudaStream_t st);
// Frames of a time-lapse chunk unless the caller names them. An eighth of the stack, in 2 to
// 32 MiB: only the first upload and the last download overlap nothing, and a chunk's copies stay
// long against its launches (24 frames of 512x512, 11x11 NRMSE: 1182 us in one chunk, 804 in
// chunks). 32 MiB where the output is pageable memory: the host waits for every download to such, and
// many small ones cost more than the overlap gives (3.3 ms in eighths and 2.7 in one; pageable input
// alone 1.6 and 2.0).
inline size_t stack_chunk(size_t frames, size_t plane, bool pageable_out) {
  size_t bytes = (size_t)32 << 20;
  if (!pageable_out) bytes = std::min<size_t>(std::max<size_t>(frames * plane / 2, (size_t)2 << 20), bytes);
  return bytes / (plane * sizeof(float));
}
// One pass over the interior of every plane (where mask > 0, if there is one), with
// the range mm_in of its values; mm_out (or null) receives the range of the results;
// shared_range: one range for all planes (the interior slices of a volume).
// Normalisation (java/Utils.java:985-1031) is kPassRange and kPassRemap.
enum PlanePass {
  kPassRange,        // the range alone
  kPassRemap,        // (v - min) / (max - min + eps) in FP32
  kPassRemapInvert,  // remap, then the NRMSE inversion (java/CLUtils.java:809-821)
  kPassMask,         // v times the mask
  kPassAbsDiff       // 1 - remap, the maximum starting at Float.MIN_VALUE (java/CLUtils.java:936-960)
};
void launch_plane_pass(PlanePass op, float* a, const float* mask, int w, int h, int rw, int rh, int planes,
                       const unsigned* mm_in, unsigned* mm_out, int num_sms, cudaStream_t st,
                       bool shared_range = false);

// gat.cu
__global__ void k_gat(float* img, size_t n, double gain, double c);
// Parameter points of one launch of the GAT objective's moments kernels
// (gain and c = 3/8 gain^2 + sigma^2 - gain offset per point).
constexpr int kGatMaxPoints = 4;
struct GatPoints {
  double gain[kGatMaxPoints], c[kGatMaxPoints];
};
__global__ void k_gat_block_moments(const float* img, int W, int bw, int bh, int nbx, GatPoints pts, double* out);
bool gat_grid(int w, int h, int* bw, int* bh, int* nbx, int* nby);
double gat_error(const double* sums, int nblocks, int bw, int bh);
__global__ void k_gat_block_moments3d(const float* vol, int W, int H, int bw, int bh, int bd, int nbx, int nby,
                                      GatPoints pts, double* out);
void gat3d_grid(int w, int h, int d, int* bw, int* bh, int* bd, int* nbx, int* nby, int* nbz);

// shape.cu (k_block_phase is declared in shape.cuh, next to PhaseRef)
__global__ void k_patch_hu(const float* img, int W, int H, Ellipse e, int patch_size, double ref_hu1, float* out,
                           float* stds_out);
__global__ void k_hu_features(const float* img, const float* means, const float* stds, int W, int bw, int bh,
                              int nx, int n, float* feat, float* sig);
__global__ void k_hu_pairs(const float* feat, const float* sig, int n, int W, int rw, int rh, int nx, float* out);
__global__ void k_phase_dft(const float* img, const float* means, const float* stds, int W, int bw, int bh, int nx,
                            int n, double* fr, double* fi);
__global__ void k_gather_interior(const float* a, int W, int rw, int rh, int nx, int n, float* out);
// The all-pairs phase map (shape.cu): one CTA per reference block, on stream st.
void launch_phase_pairs(const double* fr, const double* fi, const float* sig, int n, int bw, int bh, int W, int nx,
                        float* out, cudaStream_t st);

}  // namespace sred
