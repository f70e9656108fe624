// 3D (volume) block repetition maps: local statistics and one reference
// block against every interior block of a volume, with the host steps of
// java/CLUtils.java:1133-1637 (metric transform, relevance mask,
// normalisation) on the device.
//
// FP32 in the reference kernels' evaluation order (cl/kernelGetLocalStatistics3D.cl,
// cl/kernelGetBlock{Pearson,Ssim,Nrmse,AbsDiffStds}3D.cl); compiled with
// -fmad=false so that no multiply-add is fused. One thread per voxel, threads
// of a warp on consecutive x so that every gather of the block is coalesced;
// the block offsets (and reference voxels) sit in shared memory and the
// Pearson chain re-reads the block through L1 instead of holding it in a
// local array.
#include <float.h>

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

// Order-preserving key of a float for atomicMin/atomicMax on unsigned ints
// (-0 orders below +0, as Math.min / Math.max do).
__device__ __forceinline__ unsigned f2key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
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

template <bool CACHE>
__global__ void __launch_bounds__(128)
    k_block_map3d_t(const float* __restrict__ img, Vol3 v, const int* __restrict__ off,
                    const float* __restrict__ ref, float ref_mean, float ref_std, int metric,
                    const float* __restrict__ means, const float* __restrict__ stds, float* __restrict__ out) {
  extern __shared__ int s_off[];
  float* s_ref = reinterpret_cast<float*>(s_off + v.k);
  float* s_t = s_ref + v.k;  // CACHE: [K][128] normalised block values of the Pearson chain
  for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < v.k; i += blockDim.x * blockDim.y) {
    s_off[i] = off[i];
    s_ref[i] = ref[i];
  }
  __syncthreads();
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p)) return;
  if (!interior3(x, y, z, v)) {
    out[p] = 0.0f;
    return;
  }
  const float tstd = stds[p];
  const float* c = img + p;
  const int K = v.k;
  if (metric == kAbsDiff) {  // cl/kernelGetBlockAbsDiffStds3D.cl
    out[p] = fabsf(ref_std - tstd);
    return;
  }
  const float tmean = means[p];
  if (metric == kPearson) {
    // cl/kernelGetBlockPearson3D.cl: min-max of the block, minus its mean,
    // min-max again, then the covariance with the reference. Every division of
    // a pass shares its divisor (div_fixed: correctly rounded, as the
    // kernel's own divisions); with CACHE the first normalisation is kept in
    // shared memory for the last pass instead of being computed again.
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    float mn = FLT_MAX, mx = -FLT_MAX;
    for (int i = 0; i < K; i++) {
      const float t = c[s_off[i]];
      mn = fminf(mn, t);
      mx = fmaxf(mx, t);
    }
    const float d1 = mx - mn + kEps, y1 = __frcp_rn(d1);
    float mn2 = FLT_MAX, mx2 = -FLT_MAX;
    for (int i = 0; i < K; i++) {
      const float t = div_fixed(c[s_off[i]] - mn, d1, y1) - tmean;
      if (CACHE) s_t[i * 128 + tid] = t;
      mn2 = fminf(mn2, t);
      mx2 = fmaxf(mx2, t);
    }
    const float d2 = mx2 - mn2 + kEps, y2 = __frcp_rn(d2);
    float cov = 0.0f;
    for (int i = 0; i < K; i++) {
      const float t = CACHE ? s_t[i * 128 + tid] : div_fixed(c[s_off[i]] - mn, d1, y1) - tmean;
      cov += s_ref[i] * div_fixed(t - mn2, d2, y2);
    }
    cov /= (float)(K - 1);
    if (ref_std == 0.0f && tstd == 0.0f) out[p] = 1.0f;
    else if (ref_std == 0.0f || tstd == 0.0f) out[p] = 0.0f;
    else out[p] = fmaxf(0.0f, cov / ((ref_std * tstd) + kEps));
    return;
  }
  if (metric == kSsim) {  // cl/kernelGetBlockSsim3D.cl
    float cov = 0.0f;
    for (int i = 0; i < K; i++) cov += s_ref[i] * (c[s_off[i]] - tmean);
    cov /= (float)(K - 1);
    if (ref_std == 0.0f && tstd == 0.0f) {
      out[p] = 1.0f;
    } else if (ref_std == 0.0f || tstd == 0.0f) {
      out[p] = 0.0f;
    } else {
      const float ssim = ((2.0f * ref_mean * tmean + kC1) * (2.0f * cov + kC2)) /
                         (((ref_mean * ref_mean) + (tmean * tmean) + kC1) * ((ref_std * ref_std) + (tstd * tstd) + kC2));
      out[p] = fmaxf(0.0f, ssim);
    }
    return;
  }
  // NRMSE, cl/kernelGetBlockNrmse3D.cl
  float mse = 0.0f;
  for (int i = 0; i < K; i++) {
    const float d = s_ref[i] - (c[s_off[i]] - tmean);
    mse += d * d;
  }
  mse /= (float)K;
  out[p] = sqrtf(mse);
}

cudaError_t launch_block_map3d(const float* img, Vol3 v, const int* off, const float* ref, float ref_mean,
                               float ref_std, int metric, const float* means, const float* stds, float* out,
                               cudaStream_t st, int z1) {
  const dim3 grid((v.W + 31) / 32, (v.H + 3) / 4, (z1 < 0 ? v.D : z1) - v.z0), blk(32, 4);
  // The Pearson chain caches its first normalisation (K x 128 floats) while
  // that fits in 96 KB of shared memory; past it, it recomputes.
  const size_t smem_base = 2 * sizeof(int) * (size_t)v.k;
  const size_t smem_cache = smem_base + sizeof(float) * 128 * (size_t)v.k;
  if (metric == kPearson && smem_cache <= 96 * 1024) {
    if (smem_cache > 48 * 1024) {
      const cudaError_t e =
          cudaFuncSetAttribute(k_block_map3d_t<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cache);
      if (e != cudaSuccess) return e;
    }
    k_block_map3d_t<true><<<grid, blk, smem_cache, st>>>(img, v, off, ref, ref_mean, ref_std, metric, means, stds,
                                                         out);
  } else {
    k_block_map3d_t<false><<<grid, blk, smem_base, st>>>(img, v, off, ref, ref_mean, ref_std, metric, means, stds,
                                                          out);
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

// Host steps on the interior (java/CLUtils.java:1459-1471, 1590-1600): NRMSE
// inverted (0 -> 1), Abs-diff turned into 1 - x.
__global__ void k_block3d_post(float* __restrict__ a, Vol3 v, int metric) {
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p) || !interior3(x, y, z, v)) return;
  if (metric == kNrmse) a[p] = a[p] == 0.0f ? 1.0f : 1.0f / a[p];
  else if (metric == kAbsDiff) a[p] = 1.0f - a[p];
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

// java/Utils.java:1572-1630 (normalizeImage3D): min and max over the interior
// (where mask > 0 when a mask is given); mm = {min key, max key}. Grid-stride
// over the volume (a grid of a few CTAs per SM) so that each warp issues one
// pair of atomics for many voxels.
__global__ void k_minmax3d(const float* __restrict__ a, const float* __restrict__ mask, Vol3 v,
                           unsigned* __restrict__ mm) {
  const size_t n = (size_t)v.W * v.H * v.D, plane = (size_t)v.W * v.H;
  unsigned lo = 0xffffffffu, hi = 0u;
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(p / plane), y = (int)((p % plane) / v.W), x = (int)(p % v.W);
    if (interior3(x, y, z, v) && (!mask || mask[p] > 0.0f)) {
      const unsigned k = f2key(a[p]);
      lo = min(lo, k);
      hi = max(hi, k);
    }
  }
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0 && lo != 0xffffffffu) {
    atomicMin(mm, lo);
    atomicMax(mm + 1, hi);
  }
}

__global__ void k_remap3d(float* __restrict__ a, const float* __restrict__ mask, Vol3 v,
                          const unsigned* __restrict__ mm) {
  if (mm[0] == 0xffffffffu) return;  // no voxel selected: the reference changes nothing
  int x, y, z;
  size_t p;
  if (!voxel(v, &x, &y, &z, &p) || !interior3(x, y, z, v) || (mask && !(mask[p] > 0.0f))) return;
  const float mn = key2f(mm[0]), mx = key2f(mm[1]);
  a[p] = (a[p] - mn) / (mx - mn + kEps);
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
// a scan. Where S reaches 2^24 the thread that holds the element adds its run one by
// one in FP32 (the sum's binade rises at most 253 times), and the others continue from
// there. Subnormal sums share the lowest binade's ulp; a sum past the largest float is
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

__global__ void __launch_bounds__(kSumThreads) k_noise3d(const float* __restrict__ stds, Vol3 v,
                                                         float* __restrict__ sum) {
  extern __shared__ float s_x[];
  __shared__ Step s_warp[32];
  __shared__ float s_sum;
  __shared__ int s_next, s_total;
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
    const float* run = s_x + tid * (kSumRun + 1);
    int first = 0;  // the runs before it are in s
    while (first < kSumThreads) {
      if (!(s <= 3.402823466e38f)) {  // Inf stays, unless a NaN follows
        bool nan = s != s;
        for (int j = 0; j < kSumRun; j++) nan |= run[j] != run[j] && tid >= first;
        if (__syncthreads_or(nan)) s = nanf("");
        break;
      }
      // s = S 2^(e - 150) with e = max(1, its biased exponent); x / ulp in two exact steps
      const unsigned bits = __float_as_uint(s);
      const int e = max(1, (int)(bits >> 23));
      const int S = (bits >> 23) ? (int)((bits & 0x7fffffu) | 0x800000u) : (int)bits;
      const int up = 150 - e, u1 = min(up, 127), u2 = up - u1;  // up: -104 .. 149
      const float f1 = __uint_as_float((unsigned)(u1 + 127) << 23), f2 = __uint_as_float((unsigned)(u2 + 127) << 23);
      int sum = 0;
      bool tie = false, big = false;  // (a NaN counts as big: the FP32 additions meet it)
#pragma unroll
      for (int j = 0; j < kSumRun; j++) {
        const float t = run[j] * f1 * f2, q = rintf(t);
        big |= !(t < (float)kSumTop);
        tie |= fabsf(t - q) == 0.5f;
        sum += (int)q;
      }
      Step a{0, 0};
      if (tid >= first) a.e = a.o = big ? kSumTop : min(sum, kSumTop);
      tie = tie && !big && tid >= first;
      if (tid == 0) s_next = kSumThreads;
      Step before, after;
      if (__syncthreads_or(tie)) {
        if (tie) {
          a = Step{0, 0};
          for (int j = 0; j < kSumRun; j++) {
            const float t = run[j] * f1 * f2, fl = floorf(t), fr = t - fl;
            const int k = (int)fl;
            a = then(a, fr == 0.5f ? Step{k + (k & 1), k + !(k & 1)} : Step{k + (fr > 0.5f), k + (fr > 0.5f)});
          }
        }
        Step in = a;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const Step b = shfl_up(in, d);
          if (lane >= d) in = then(b, in);
        }
        if (lane == 31) s_warp[w] = in;
        __syncthreads();
        Step pre = s_warp[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const Step b = shfl_up(pre, d);
          if (lane >= d) pre = then(b, pre);
        }
        pre = Step{__shfl_sync(0xffffffffu, pre.e, (w + 31) & 31), __shfl_sync(0xffffffffu, pre.o, (w + 31) & 31)};
        if (w == 0) pre = Step{0, 0};
        const Step ex = shfl_up(in, 1);
        before = lane == 0 ? pre : then(pre, ex);
        after = then(pre, in);
      } else {  // one increment for both parities
        int in = a.e;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int b = __shfl_up_sync(0xffffffffu, in, d);
          if (lane >= d) in = min(in + b, kSumTop);
        }
        if (lane == 31) s_warp[w].e = in;
        __syncthreads();
        int pre = s_warp[lane].e;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int b = __shfl_up_sync(0xffffffffu, pre, d);
          if (lane >= d) pre = min(pre + b, kSumTop);
        }
        pre = __shfl_sync(0xffffffffu, pre, (w + 31) & 31);
        if (w == 0) pre = 0;
        const int ex = __shfl_up_sync(0xffffffffu, in, 1);
        before.e = before.o = lane == 0 ? pre : min(pre + ex, kSumTop);
        after.e = after.o = min(pre + in, kSumTop);
      }
      const int s0 = S + ((S & 1) ? before.o : before.e), s1 = S + ((S & 1) ? after.o : after.e);
      if (s0 < kSumTop && s1 >= kSumTop) {  // at most one thread: the binade ends in its run
        float t = (float)s0;
        t = u2 ? t / f2 / f1 : t / f1;
#pragma unroll
        for (int j = 0; j < kSumRun; j++) t += run[j];
        s_sum = t;
        s_next = tid + 1;
      }
      if (tid == kSumThreads - 1) s_total = s1;
      __syncthreads();
      first = s_next;
      if (s_total < kSumTop) {
        const float t = (float)s_total;
        s = u2 ? t / f2 / f1 : t / f1;
      } else {
        s = s_sum;
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
