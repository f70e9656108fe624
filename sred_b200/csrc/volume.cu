// 3D (volume) block repetition maps: local statistics and one reference
// block against every interior block of a volume, with the host steps of
// java/CLUtils.java:1133-1637 (metric transform, relevance mask,
// normalisation) on the device.
//
// FP32 in the reference kernels' evaluation order (cl/kernelGetLocalStatistics3D.cl,
// cl/kernelGetBlock{Pearson,Ssim,Nrmse,AbsDiffStds}3D.cl); compiled with
// -fmad=false so that no multiply-add is fused.
#include <float.h>

#include <algorithm>
#include <type_traits>

#include "ranges.cuh"
#include "volume.cuh"

namespace sred {

namespace {

__device__ __forceinline__ bool interior3(int x, int y, int z, const Vol3& v) {
  return x >= v.rw && x < v.W - v.rw && y >= v.rh && y < v.H - v.rh && z >= v.rd && z < v.D - v.rd;
}

// Voxel of this thread for the (32, 4) block and ((W+31)/32, (H+3)/4, D) grid
// (or a grid of fewer slices starting at slice v.z0).
__device__ __forceinline__ bool voxel(const Vol3& v, int* x, int* y, int* z, size_t* p) {
  *x = blockIdx.x * blockDim.x + threadIdx.x;
  *y = blockIdx.y * blockDim.y + threadIdx.y;
  *z = blockIdx.z + v.z0;
  if (*x >= v.W || *y >= v.H) return false;
  *p = ((size_t)*z * v.H + *y) * v.W + *x;
  return true;
}

}  // namespace

__global__ void __launch_bounds__(128)
    k_local_stats3d(const float* __restrict__ img, Vol3 v, const int* __restrict__ off, float* __restrict__ means,
                    float* __restrict__ stds) {
  extern __shared__ int s_off[];
  for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < v.k; i += blockDim.x * blockDim.y) s_off[i] = off[i];
  __syncthreads();
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p)) return;
  if (!interior3(x, y, z, v)) {
    means[p] = 0.0f;
    stds[p] = 0.0f;
    return;
  }
  const float* c = img + p;
  const int K = v.k;
  float mean = 0.0f;
  for (int i = 0; i < K; i++) mean += c[s_off[i]];
  mean /= (float)K;
  float var = 0.0f;
  for (int i = 0; i < K; i++) {
    const float d = c[s_off[i]] - mean;
    var += d * d;
  }
  means[p] = mean;
  stds[p] = sqrtf(var / (float)(K - 1));
}

// ---------------------------------------------------------------------------
// The block map. A thread takes PX voxels of a row; neighbours share all but one
// value of each row of the block, so a window of PX values slides along it: one load
// (through L1) serves PX voxels, and an element's offset and reference value are
// fetched once for PX. The local statistics are the first sweeps of the same kernel,
// the metric transform and the range its last step, and Pearson's first normalisation
// is computed again in the last sweep (five operations) rather than kept.
// Bound by FP32 issue, 24 operations an element and voxel for Pearson: 199 us for
// 256x256x64, 5x5x5 (33 elements), normalised, where one voxel a thread in four
// kernels took 330.
// ---------------------------------------------------------------------------
namespace {

// Visits the block in the reference's order: f(i, w), w(q) the value of voxel column q.
// A window at the end of a row holds values of the next one, which only discarded voxels
// see; with LAST (the slice whose blocks reach the end of the volume) it repeats the row's
// last value instead. room: columns from the first voxel to the last of the row.
template <int PX, bool LAST, class F>
__device__ __forceinline__ void sweep3(const float* c, const int2* rows, int nrows, int room, F f) {
  int i = 0;
  for (int r = 0; r < nrows; r++) {
    const int2 row = rows[r];  // offset of its first voxel, voxels (odd)
    const float* p = c + row.x;
    int n = row.y, last = room + (n >> 1);
    float w[PX];
#pragma unroll
    for (int q = 0; q < PX - 1; q++) w[q] = p[LAST ? min(q, last) : q];
    auto element = [&](auto jc) {
      constexpr int j = decltype(jc)::value;
      w[(j + PX - 1) % PX] = p[LAST ? min(j + PX - 1, last) : j + PX - 1];
      f(i + j, [&](int q) { return w[(j + q) % PX]; });
    };
    for (; n >= 4; n -= 4, i += 4, p += 4, last -= 4) {
      element(std::integral_constant<int, 0>());
      element(std::integral_constant<int, 1>());
      element(std::integral_constant<int, 2>());
      element(std::integral_constant<int, 3>());
    }
    element(std::integral_constant<int, 0>());
    if (n == 3) {
      element(std::integral_constant<int, 1>());
      element(std::integral_constant<int, 2>());
    }
    i += n;
  }
}

constexpr int kRows3 = 8;  // rows of a CTA, one warp each

// The voxels x .. x + PX - 1 (of which those right of the interior are discarded): their
// values, local stds and range.
template <int METRIC, int PX, bool LAST>
__device__ __forceinline__ void map_voxels(const float* c, int x, const Vol3& v, const int2* rows, const float* s_ref,
                                           float ref_mean, float ref_std, float (&val)[PX], float (&sd)[PX],
                                           unsigned& lo, unsigned& hi) {
  const int K = v.k, room = v.W - 1 - x;
  float mean[PX], var[PX], acc[PX], mn[PX], mx[PX];
#pragma unroll
  for (int q = 0; q < PX; q++) {
    mean[q] = var[q] = acc[q] = 0.0f;
    mn[q] = FLT_MAX;
    mx[q] = -FLT_MAX;
  }
  sweep3<PX, LAST>(c, rows, v.nrows, room, [&](int, auto w) {
#pragma unroll
    for (int q = 0; q < PX; q++) {
      mean[q] += w(q);
      if (METRIC == kPearson) {
        mn[q] = fminf(mn[q], w(q));
        mx[q] = fmaxf(mx[q], w(q));
      }
    }
  });
  // cl/kernelGetBlockPearson3D.cl: min-max of the block, minus its mean, min-max
  // again, then the covariance with the reference. Every division of a sweep shares
  // its divisor (div_fixed: correctly rounded, as the kernel's own divisions).
  float d1[PX], y1[PX], mn2[PX], mx2[PX];
#pragma unroll
  for (int q = 0; q < PX; q++) {
    mean[q] /= (float)K;
    d1[q] = mx[q] - mn[q] + kEps;
    y1[q] = METRIC == kPearson ? __frcp_rn(d1[q]) : 0.0f;
    mn2[q] = FLT_MAX;
    mx2[q] = -FLT_MAX;
  }
  sweep3<PX, LAST>(c, rows, v.nrows, room, [&](int i, auto w) {
    const float rf = METRIC == kSsim || METRIC == kNrmse ? s_ref[i] : 0.0f;
#pragma unroll
    for (int q = 0; q < PX; q++) {
      const float d = w(q) - mean[q];
      var[q] += d * d;
      if (METRIC == kPearson) {
        const float t = div_fixed(w(q) - mn[q], d1[q], y1[q]) - mean[q];
        mn2[q] = fminf(mn2[q], t);
        mx2[q] = fmaxf(mx2[q], t);
      } else if (METRIC == kSsim) {  // cl/kernelGetBlockSsim3D.cl
        acc[q] += rf * d;
      } else if (METRIC == kNrmse) {  // cl/kernelGetBlockNrmse3D.cl
        const float e = rf - d;
        acc[q] += e * e;
      }
    }
  });
  if (METRIC == kPearson) {
#pragma unroll
    for (int q = 0; q < PX; q++) {
      mx2[q] = mx2[q] - mn2[q] + kEps;
      mx[q] = __frcp_rn(mx2[q]);
    }
    sweep3<PX, LAST>(c, rows, v.nrows, room, [&](int i, auto w) {
      const float rf = s_ref[i];
#pragma unroll
      for (int q = 0; q < PX; q++) {
        const float t = div_fixed(w(q) - mn[q], d1[q], y1[q]) - mean[q];
        acc[q] += rf * div_fixed(t - mn2[q], mx2[q], mx[q]);
      }
    });
  }
#pragma unroll
  for (int q = 0; q < PX; q++) {
    if (x + q >= v.W - v.rw) break;
    const float s = sqrtf(var[q] / (float)(K - 1));
    float o;
    if (METRIC == kAbsDiff) {  // cl/kernelGetBlockAbsDiffStds3D.cl, java/CLUtils.java:1590-1600
      o = 1.0f - fabsf(ref_std - s);
    } else if (METRIC == kNrmse) {  // java/CLUtils.java:1459-1471
      o = sqrtf(acc[q] / (float)K);
      o = o == 0.0f ? 1.0f : 1.0f / o;
    } else if (ref_std == 0.0f && s == 0.0f) {
      o = 1.0f;
    } else if (ref_std == 0.0f || s == 0.0f) {
      o = 0.0f;
    } else if (METRIC == kPearson) {
      o = fmaxf(0.0f, acc[q] / (float)(K - 1) / ((ref_std * s) + kEps));
    } else {
      const float cov = acc[q] / (float)(K - 1);
      o = fmaxf(0.0f, ((2.0f * ref_mean * mean[q] + kC1) * (2.0f * cov + kC2)) /
                          (((ref_mean * ref_mean) + (mean[q] * mean[q]) + kC1) *
                           ((ref_std * ref_std) + (s * s) + kC2)));
    }
    val[q] = o;
    sd[q] = s;
    lo = min(lo, ord_bits(o));
    hi = max(hi, ord_bits(o));
  }
}

template <int METRIC, int PX>
__global__ void __launch_bounds__(32 * kRows3)
    k_block_map3d(const float* __restrict__ img, Vol3 v, const int* __restrict__ off, const float* __restrict__ ref,
                  float ref_mean, float ref_std, float* __restrict__ out, float* __restrict__ stds,
                  unsigned* __restrict__ mm) {
  extern __shared__ int2 s_rows[];
  float* s_ref = reinterpret_cast<float*>(s_rows + v.nrows);
  const int2* rows = reinterpret_cast<const int2*>(off + v.k + (v.k & 1));
  for (int i = threadIdx.x; i < v.nrows; i += 32 * kRows3) s_rows[i] = rows[i];
  for (int i = threadIdx.x; i < v.k; i += 32 * kRows3) s_ref[i] = ref[i];
  __syncthreads();
  // the tiles start at the first interior column; the first one also owns those before it
  const int lane = threadIdx.x & 31, x0 = v.rw + blockIdx.x * 32 * PX, x = x0 + lane * PX;
  const int y = blockIdx.y * kRows3 + (threadIdx.x >> 5), z = blockIdx.z + v.z0;
  const size_t base = ((size_t)z * v.H + y) * v.W;
  unsigned lo = 0xffffffffu, hi = 0u;
  float val[PX], sd[PX];
#pragma unroll
  for (int q = 0; q < PX; q++) val[q] = sd[q] = 0.0f;
  if (interior3(x, y, z, v)) {
    if (z == v.D - 1 - v.rd)
      map_voxels<METRIC, PX, true>(img + base + x, x, v, s_rows, s_ref, ref_mean, ref_std, val, sd, lo, hi);
    else
      map_voxels<METRIC, PX, false>(img + base + x, x, v, s_rows, s_ref, ref_mean, ref_std, val, sd, lo, hi);
  }
  if (y < v.H) {
#pragma unroll
    for (int q = 0; q < PX; q++)
      if (x + q < v.W) {
        out[base + x + q] = val[q];
        if (stds) stds[base + x + q] = sd[q];
      }
    if (blockIdx.x == 0)
      for (int i = lane; i < min(v.rw, v.W); i += 32) {
        out[base + i] = 0.0f;
        if (stds) stds[base + i] = 0.0f;
      }
  }
  if (mm) cta_minmax(lo, hi, mm);
}

template <int METRIC>
void launch_map3d(const float* img, const Vol3& v, const int* off, const float* ref, float ref_mean, float ref_std,
                  float* out, float* stds, unsigned* mm, cudaStream_t st, int slices) {
  const size_t smem = sizeof(int2) * v.nrows + sizeof(float) * v.k;
  const int iw = v.W - 2 * v.rw;
  auto run = [&](auto kernel, int px) {
    const dim3 grid(std::max(1, (v.W - v.rw + 32 * px - 1) / (32 * px)), (v.H + kRows3 - 1) / kRows3, slices);
    kernel<<<grid, 32 * kRows3, smem, st>>>(img, v, off, ref, ref_mean, ref_std, out, stds, mm);
  };
  // the widest window whose warps the interior fills at least half
  if (iw > 64) run(k_block_map3d<METRIC, 4>, 4);
  else if (iw > 32) run(k_block_map3d<METRIC, 2>, 2);
  else run(k_block_map3d<METRIC, 1>, 1);
}

}  // namespace

cudaError_t launch_block_map3d(const float* img, Vol3 v, const int* off, const float* ref, float ref_mean,
                               float ref_std, int metric, float* out, float* stds, unsigned* mm, cudaStream_t st,
                               int z1) {
  const int n = z1 - v.z0;
  switch (metric) {
    case kPearson: launch_map3d<kPearson>(img, v, off, ref, ref_mean, ref_std, out, stds, mm, st, n); break;
    case kSsim: launch_map3d<kSsim>(img, v, off, ref, ref_mean, ref_std, out, stds, mm, st, n); break;
    case kNrmse: launch_map3d<kNrmse>(img, v, off, ref, ref_mean, ref_std, out, stds, mm, st, n); break;
    default: launch_map3d<kAbsDiff>(img, v, off, ref, ref_mean, ref_std, out, stds, mm, st, n); break;
  }
  return cudaGetLastError();
}

// Elementwise a[i] / b by div_fixed (diagnostics: checked against IEEE division).
__global__ void k_divide_fixed(const float* __restrict__ a, size_t n, float b, float* __restrict__ out) {
  const float y = __frcp_rn(b);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = div_fixed(a[i], b, y);
}

// Elementwise a[i] / b by the FP64 div_fixed (diagnostics: checked against IEEE division).
__global__ void k_divide_fixed64(const double* __restrict__ a, size_t n, double b, double* __restrict__ out) {
  const double y = __drcp_rn(b);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = div_fixed(a[i], b, y);
}

// java/Utils.java:1501-1525 (getRelevanceMask3D) for the threshold
// noise_var * c; map (if not null) is multiplied by the mask (applyMask3D).
__global__ void k_mask3d(const float* __restrict__ stds, Vol3 v, float thr, float* __restrict__ mask,
                         float* __restrict__ map) {
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p)) return;
  float m = 0.0f;
  if (interior3(x, y, z, v)) m = (stds[p] * stds[p]) <= thr ? 0.0f : 1.0f;
  mask[p] = m;
  if (map) map[p] *= m;
}

// ---------------------------------------------------------------------------
// 3D global repetition map: flags, operand packing and finalisation around
// the 2D pair engines (cl/kernelGetGlobal*3D.cl, java/CLUtils.java:2225-2790).
// ---------------------------------------------------------------------------

// mask: sigma^2 > threshold on the interior (getRelevanceMask3D).
// flags: 1 = reference and test block (interior, !(sigma^2 < threshold),
// sigma^2 != 0: the 3D kernels skip a reference voxel of zero variance);
// 2 = test block only, sigma == 0 (a flat block still counts as a test block
// of Pearson, SSIM and NRMSE; flat_columns = 0 drops it, as Abs-diff does).
// A voxel with sigma != 0 but sigma^2 == 0 (sigma below 1.1e-23) is neither;
// the reference would still use it as a test block.
// n_mask counts mask > 0 (the command's nPixels).
__global__ void k_flags3d(const float* __restrict__ stds, Vol3 v, float thr, int flat_columns,
                          float* __restrict__ mask, uint8_t* __restrict__ flags,
                          unsigned long long* __restrict__ n_mask) {
  const size_t n = (size_t)v.W * v.H * v.D, plane = (size_t)v.W * v.H;
  unsigned c = 0;
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(p / plane), y = (int)((p % plane) / v.W), x = (int)(p % v.W);
    const bool in = interior3(x, y, z, v);
    const float s = stds[p];
    const float s2 = s * s;
    const float m = (in && !(s2 <= thr)) ? 1.0f : 0.0f;
    mask[p] = m;
    uint8_t f = 0;
    if (in && !(s2 < thr)) {
      if (s2 != 0.0f) f = 1;
      else if (s == 0.0f && flat_columns) f = 2;
    }
    flags[p] = f;
    c += m > 0.0f ? 1u : 0u;
  }
  const unsigned wc = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && wc) atomicAdd(n_mask, (unsigned long long)wc);
}

// num / (den nPixels + eps) in FP64 over the interior, with the flat test
// blocks' closed-form share: n_flat pairs of weight 2^-(a_p^2) each, and for
// NRMSE a term sqrt((K-1)/K) sigma_p per pair times that weight (the flat
// block's centred vector is zero). NRMSE and Abs-diff are then inverted where
// mask > 0 (the FP32 value; 0 -> 1), and the mask applied when apply_mask.
__global__ void k_finalize3d(const int* __restrict__ slot, Vol3 v, const double* __restrict__ num,
                             const double* __restrict__ den, const BlockParams* __restrict__ params, int n_flat,
                             int metric, double sk, double n_pixels, const float* __restrict__ mask, int apply_mask,
                             float* __restrict__ out) {
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p)) return;
  float o = 0.0f;
  if (interior3(x, y, z, v)) {
    const int s = slot[p];
    double nu = 0.0, de = 0.0;
    if (s >= 0) {
      const BlockParams bp = params[s];
      const double a = (double)bp.a;
      const double w0 = exp2(-(a * a));
      nu = num[s];
      de = den[s] + (double)n_flat * w0;
      if (metric == kNrmse) nu += (double)n_flat * sk * (double)bp.sigma * w0;
    }
    o = (float)(nu / (de * n_pixels + (double)kEps));
    if ((metric == kNrmse || metric == kAbsDiff) && mask[p] > 0.0f) o = (o == 0.0f) ? 1.0f : 1.0f / o;
    if (apply_mask) o *= mask[p];
  }
  out[p] = o;
}

int build_ellipsoid(int bw, int bh, int bd, int W, int H, int* off) {
  const int rw = bw / 2, rh = bh / 2, rd = bd / 2;
  int k = 0;
  for (int z = -rd; z <= rd; z++)
    for (int y = -rh; y <= rh; y++)
      for (int x = -rw; x <= rw; x++) {
        const float fx = (float)x, fy = (float)y, fz = (float)z;
        if (((fx * fx) / (float)(rw * rw)) + ((fy * fy) / (float)(rh * rh)) + ((fz * fz) / (float)(rd * rd)) <=
            1.0f) {
          if (off && k < kMaxK3) off[k] = z * W * H + y * W + x;
          k++;
        }
      }
  return k;
}

// ---------------------------------------------------------------------------
// Noise variance of a volume: the sum of sigma^2 over the interior in raster order,
// every partial sum rounded to FP32 (java/Utils.java:1467-1483). One CTA.
//
// While the sum s stays within a binade, s = S ulp with a whole S < 2^24, and adding x
// adds the whole number nearest to x / ulp; a tie goes by the parity of S. An element,
// and any run of elements, is then a function of S's parity: two whole increments, and
// those compose associatively. So 16,384 elements at a time are 1,024 threads' runs and
// a scan of the warps' sums. Where S reaches 2^24 the warp that holds the element steps
// through its 512 by itself, the run that ends the binade in FP32 (the binade rises at
// most 253 times), and the others continue from there. Subnormal sums share the lowest binade's ulp; a sum past the largest float is
// Inf or NaN for good. Bound by the one SM's issue slots: 0.26 ms for
// 128x128x48 (676,000 elements), where the copy to the host and the serial sum there
// added 1.0 ms to the map.
// ---------------------------------------------------------------------------
namespace {

constexpr int kSumThreads = 1024, kSumRun = 16, kSumChunk = kSumThreads * kSumRun;
constexpr int kSumSmem = (kSumChunk + kSumChunk / kSumRun) * (int)sizeof(float);  // runs 17 floats apart
constexpr int kSumTop = 1 << 24;

// Increments for an even and an odd sum; past kSumTop only "at least" matters.
struct Step {
  int e, o;
};
__device__ __forceinline__ Step then(Step a, Step b) {
  Step r;
  r.e = min(a.e + ((a.e & 1) ? b.o : b.e), kSumTop);
  r.o = min(a.o + ((a.o & 1) ? b.e : b.o), kSumTop);
  return r;
}
__device__ __forceinline__ Step shfl_up(Step a, int d) {
  return Step{__shfl_up_sync(0xffffffffu, a.e, d), __shfl_up_sync(0xffffffffu, a.o, d)};
}

// s = S ulp with a whole S (below kSumTop unless s is not finite), x / ulp in two exact
// steps of f1 and f2: ulp = 2^(e - 150) for e = max(1, the biased exponent of s).
struct Grid {
  int S;
  float f1, f2;
  __device__ __forceinline__ explicit Grid(float s) {
    const unsigned bits = __float_as_uint(s);
    const int e = max(1, (int)(bits >> 23)), up = 150 - e, u1 = min(up, 127);  // up: -104 .. 149
    S = (bits >> 23) ? (int)((bits & 0x7fffffu) | 0x800000u) : (int)bits;
    f1 = __uint_as_float((unsigned)(u1 + 127) << 23);
    f2 = __uint_as_float((unsigned)(up - u1 + 127) << 23);
  }
  __device__ __forceinline__ float at(int n) const { return (float)n / f2 / f1; }
};

// A run's increment where no element ties or rounds to 2^22 ulp or more; with one that does,
// or a NaN, *odd is set and run_steps gives it. Rounds by adding 1.5 2^23 (conversions issue
// at an eighth of the rate); from 2^22 - 0.5 on that sum is 2^24, past the low 23 bits.
__device__ __forceinline__ int run_increment(const float* run, const Grid& g, bool* odd) {
  const float magic = 12582912.0f;
  int sum = 0;
  bool o = false;
#pragma unroll
  for (int j = 0; j < kSumRun; j++) {
    const float t = run[j] * g.f1 * g.f2, m = t + magic;
    o |= !(t < 4194303.5f) || fabsf(t - (m - magic)) == 0.5f;
    sum += (int)(__float_as_uint(m) & 0x7fffffu);
  }
  *odd = o;
  return sum - kSumRun * 0x400000;
}
__device__ __noinline__ Step run_steps(const float* run, float f1, float f2) {
  Step a{0, 0};
  for (int j = 0; j < kSumRun; j++) {
    const float t = run[j] * f1 * f2, fl = floorf(t), fr = t - fl;
    if (!(t < (float)kSumTop)) return Step{kSumTop, kSumTop};  // (a NaN too: the FP32 additions meet it)
    const int k = (int)fl;
    a = then(a, fr == 0.5f ? Step{k + (k & 1), k + !(k & 1)} : Step{k + (fr > 0.5f), k + (fr > 0.5f)});
  }
  return a;
}
// Inclusive composition over the lanes.
__device__ __forceinline__ Step scan_steps(Step a, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Step b = shfl_up(a, d);
    if (lane >= d) a = then(b, a);
  }
  return a;
}

// The sum after a warp's 32 runs: lanes' increments while the binade lasts, and the run
// that ends it in FP32.
__device__ float warp_sum(float s, const float* run, int lane) {
  for (int first = 0; first < 32;) {
    if (!(s <= 3.402823466e38f)) {  // Inf stays, unless a NaN follows
      bool nan = s != s;
      for (int j = 0; j < kSumRun; j++) nan |= run[j] != run[j] && lane >= first;
      return __any_sync(0xffffffffu, nan) ? nanf("") : s;
    }
    const Grid g(s);
    bool tie;
    Step a;
    a.e = a.o = run_increment(run, g, &tie);
    if (tie) a = run_steps(run, g.f1, g.f2);
    if (lane < first) a = Step{0, 0};
    a = scan_steps(a, lane);
    const int end = g.S + ((g.S & 1) ? a.o : a.e);
    const unsigned past = __ballot_sync(0xffffffffu, end >= kSumTop);
    int begin = __shfl_up_sync(0xffffffffu, end, 1);
    if (lane == 0) begin = g.S;
    if (!past) return g.at(__shfl_sync(0xffffffffu, end, 31));
    first = __ffs(past);
    float t = g.at(begin);
    if (lane == first - 1) {
#pragma unroll
      for (int j = 0; j < kSumRun; j++) t += run[j];
    }
    s = __shfl_sync(0xffffffffu, t, first - 1);
  }
  return s;
}

__global__ void __launch_bounds__(kSumThreads) k_noise3d(const float* __restrict__ stds, Vol3 v,
                                                         float* __restrict__ sum) {
  extern __shared__ float s_x[];
  __shared__ Step s_warp[32];
  __shared__ float s_sum;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned iw = v.W - 2 * v.rw, ih = v.H - 2 * v.rh;
  const size_t n = (size_t)iw * ih * (v.D - 2 * v.rd);
  // this thread's element of each row of 1,024, its address, and the step to the next row
  unsigned x = tid % iw, y = tid / iw % ih;
  const size_t wrap_y = v.W - iw, wrap_z = (size_t)(v.H - ih) * v.W;
  const unsigned dx = kSumThreads % iw, dy = kSumThreads / iw % ih, dz = kSumThreads / iw / ih;
  const size_t dq = ((size_t)dz * v.H + dy) * v.W + dx;
  size_t at = tid;
  const float* q = stds + ((size_t)(tid / iw / ih + v.rd) * v.H + y + v.rh) * v.W + x + v.rw;
  float next[kSumRun];
  auto load = [&]() {
#pragma unroll
    for (int j = 0; j < kSumRun; j++) {
      next[j] = at < n ? *q : 0.0f;
      at += kSumThreads;
      x += dx;
      y += dy;
      q += dq;
      if (x >= iw) x -= iw, y++, q += wrap_y;
      if (y >= ih) y -= ih, q += wrap_z;
    }
  };
  load();
  float s = 0.0f;
  const float* run = s_x + tid * (kSumRun + 1);
  const size_t chunks = (n + kSumChunk - 1) / kSumChunk;
  for (size_t c = 0; c < chunks; c++) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSumRun; j++) {
      const int i = j * kSumThreads + tid;
      s_x[i + i / kSumRun] = next[j] * next[j];
    }
    __syncthreads();
    if (c + 1 < chunks) load();
    int first = 0;  // the warps before it are in s
    if (c == 0) {   // half of the binades end in the first warp's 512 elements
      if (w == 0) {
        const float t = warp_sum(0.0f, run, lane);
        if (lane == 0) s_sum = t;
      }
      __syncthreads();
      s = s_sum;
      first = 1;
    }
    while (first < 32) {
      if (!(s <= 3.402823466e38f)) {
        bool nan = s != s;
        for (int j = 0; j < kSumRun; j++) nan |= run[j] != run[j] && w >= first;
        if (__syncthreads_or(nan)) s = nanf("");
        break;
      }
      const Grid g(s);
      bool tie;
      Step a;
      a.e = a.o = run_increment(run, g, &tie);
      if (w < first) {
        a = Step{0, 0};
        tie = false;
      }
      Step all;  // after warp `lane`
      if (__syncthreads_or(tie)) {
        if (tie) a = run_steps(run, g.f1, g.f2);
        a = scan_steps(a, lane);
        if (lane == 31) s_warp[w] = a;
        __syncthreads();
        all = scan_steps(s_warp[lane], lane);
      } else {  // one increment for both parities
        const int t = __reduce_add_sync(0xffffffffu, a.e);  // below 2^31
        if (lane == 0) s_warp[w].e = min(t, kSumTop);
        __syncthreads();
        int in = s_warp[lane].e;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int b = __shfl_up_sync(0xffffffffu, in, d);
          if (lane >= d) in = min(in + b, kSumTop);
        }
        all.e = all.o = in;
      }
      const int end = g.S + ((g.S & 1) ? all.o : all.e);
      const unsigned past = __ballot_sync(0xffffffffu, end >= kSumTop);
      if (past) {
        const int hit = __ffs(past) - 1;  // the binade ends in this warp
        int begin = __shfl_sync(0xffffffffu, end, max(hit - 1, 0));
        if (hit == 0) begin = g.S;
        if (w == hit) {
          const float t = warp_sum(g.at(begin), run, lane);
          if (lane == 0) s_sum = t;
        }
        __syncthreads();
        s = s_sum;
        first = hit + 1;
      } else {
        s = g.at(__shfl_sync(0xffffffffu, end, 31));
        first = 32;
      }
      __syncthreads();
    }
    if (s != s) break;
  }
  if (tid == 0) *sum = s;
}

}  // namespace

cudaError_t launch_noise3d(const float* stds, Vol3 v, float* sum, cudaStream_t st) {
  if (v.W <= 2 * v.rw || v.H <= 2 * v.rh || v.D <= 2 * v.rd) return cudaMemsetAsync(sum, 0, sizeof(float), st);
  const cudaError_t e = cudaFuncSetAttribute(k_noise3d, cudaFuncAttributeMaxDynamicSharedMemorySize, kSumSmem);
  if (e != cudaSuccess) return e;
  k_noise3d<<<1, kSumThreads, kSumSmem, st>>>(stds, v, sum);
  return cudaGetLastError();
}

}  // namespace sred
