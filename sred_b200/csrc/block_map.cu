// Block ("local") repetition map: one reference block against every interior
// block of an image (or of each frame of a stack).
//
// One streaming pass per pixel fuses the block moments with the metric: the
// kernel reads only the image and writes only the map (plus, optionally, the
// local stds the relevance mask needs). The moments and the metric follow the
// reference kernels' FP32 evaluation order with explicitly rounded operations,
// so the raw map equals the reference's (cl/kernelGetBlock{Pearson,Ssim,
// Nrmse,AbsDiffStds}2D.cl, with cl/kernelGetLocalStatistics2D.cl for the
// moments) bit for bit. The image tile and its halo are staged in shared
// memory so every pixel is read from HBM once.
//
// The host steps that follow (java/CLUtils.java:788-821, 936-960, and the
// normalisation) are one read-modify-write pass each, k_plane_pass: the range a
// pass needs is taken by the kernel that wrote the values.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "ranges.cuh"

namespace sred {

namespace {

constexpr int kThreadsY = 8;         // thread rows of a CTA (one warp each)
constexpr int kTileY = 2 * kThreadsY;  // a thread's pixels: rows y and y + 8 of the tile

using f2 = unsigned long long;  // two floats: rows y (low) and y + 8

__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The rounded product, as a b + nz with nz = (-0, -0) a kernel argument: the
// compiler merges a packed multiplication, or a multiply-add of a -0 that it can
// see, with the addition that follows into one rounding, even with .rn on both.
__device__ __forceinline__ f2 mul2(f2 a, f2 b, f2 nz) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
  return r;
}
constexpr f2 kNegZero2 = 0x8000000080000000ull;
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float* a, float* b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(v));
}

// The metric of one pixel from its block sums (reference order, explicitly
// rounded), and its local std.
__device__ __forceinline__ float block_metric_value(int metric, int K, float mean, float v, float acc, float rr,
                                                    float xx, float ref_mean, float ref_std, float* sd_out) {
  const float sd = __fsqrt_rn(__fdiv_rn(v, (float)(K - 1)));
  *sd_out = sd;
  if (metric == kAbsDiff) return fabsf(__fsub_rn(ref_std, sd));
  if (metric == kNrmse) return __fsqrt_rn(__fdiv_rn(acc, (float)K));
  if (metric == kCosine) return __fdiv_rn(acc, __fadd_rn(__fmul_rn(__fsqrt_rn(rr), __fsqrt_rn(xx)), kEps));
  const float cov = __fdiv_rn(acc, (float)(K - 1));
  if (ref_std == 0.0f && sd == 0.0f) return 1.0f;
  if (ref_std == 0.0f || sd == 0.0f) return 0.0f;
  if (metric == kPearson) return fmaxf(0.0f, __fdiv_rn(cov, __fadd_rn(__fmul_rn(ref_std, sd), kEps)));
  // SSIM, textbook sum form (cl/kernelGetBlockSsim2D.cl:79)
  const float a = __fadd_rn(__fmul_rn(__fmul_rn(2.0f, ref_mean), mean), kC1);
  const float b = __fadd_rn(__fmul_rn(2.0f, cov), kC2);
  const float cc = __fadd_rn(__fadd_rn(__fmul_rn(ref_mean, ref_mean), __fmul_rn(mean, mean)), kC1);
  const float dd = __fadd_rn(__fadd_rn(__fmul_rn(ref_std, ref_std), __fmul_rn(sd, sd)), kC2);
  return fmaxf(0.0f, __fdiv_rn(__fmul_rn(a, b), __fmul_rn(cc, dd)));
}

// The ellipse by rows: row r holds the columns -hw[r] .. hw[r]; the first and the last
// `single` rows hold one element each.
struct BlockRows {
  int k, rw, rh, single;
  short hw[kMaxK];
};

// Visits the block of a thread's 2 PX pixels in the reference's order: f(i, w)
// for element i with w(q) the value pair of pixel column q. Neighbouring pixels
// share all but one value of an element, so a window of PX pairs slides along
// each row: one shared-memory load an element for 2 PX pixels. Column c of the
// tile lies at (c % PX) p + c / PX, which keeps the loads of a warp contiguous.
// The rows of one element, most of a narrow block's, take a loop without a window
// (3x101 at 1024x1024, PX = 1: 160 us without it, 96 so).
template <int PX, class F>
__device__ __forceinline__ void sweep(const f2* base, int p, int pitch, const BlockRows& e, F f) {
  int i = 0;
  auto single = [&]() {
    int o[PX];
#pragma unroll
    for (int q = 0; q < PX; q++) o[q] = ((e.rw + q) % PX) * p + (e.rw + q) / PX;
#pragma unroll 4
    for (int r = 0; r < e.single; r++, i++, base += pitch) {
      f2 w[PX];
#pragma unroll
      for (int q = 0; q < PX; q++) w[q] = base[o[q]];
      f(i, [&](int q) { return w[q]; });
    }
  };
  single();
  for (int r = e.single; r <= 2 * e.rh - e.single; r++, base += pitch) {
    const int hw = e.hw[r], s = e.rw - hw;
    int o[4];
#pragma unroll
    for (int q = 0; q < 4; q++) o[q] = ((s + q) % PX) * p + (s + q) / PX;
    f2 w[PX];
#pragma unroll
    for (int q = 0; q < PX - 1; q++) w[q] = base[o[q]];
    auto element = [&](auto jc) {
      constexpr int j = decltype(jc)::value;
      constexpr int c = PX - 1 + j;  // the column that enters the window
      w[c % PX] = base[o[c & 3] + (c >> 2) * (4 / PX)];
      f(i + j, [&](int q) { return w[(j + q) % PX]; });
    };
    int n = 2 * hw + 1;
    for (; n >= 4; n -= 4, i += 4) {
      element(std::integral_constant<int, 0>());
      element(std::integral_constant<int, 1>());
      element(std::integral_constant<int, 2>());
      element(std::integral_constant<int, 3>());
#pragma unroll
      for (int q = 0; q < 4; q++) o[q] += 4 / PX;
    }
    // (n is odd: 1 or 3 left)
    element(std::integral_constant<int, 0>());
    if (n == 3) {
      element(std::integral_constant<int, 1>());
      element(std::integral_constant<int, 2>());
    }
    i += n;
  }
  single();
}

// The tile of PX: columns, values per column class, f2 per row.
template <int PX>
struct Tile {
  static constexpr int kX = 32 * PX;
  __host__ __device__ static int cols(int rw) { return kX + 2 * rw; }
  // p = 4 mod 8: the classes of neighbouring columns fall on different banks
  __host__ __device__ static int p(int rw) { return PX == 1 ? cols(rw) : ((cols(rw) + PX - 1) / PX + 11) / 8 * 8 - 4; }
  __host__ __device__ static int pitch(int rw) { return PX * p(rw); }
  static size_t smem(int rw, int rh, int k) {
    return sizeof(f2) * ((size_t)pitch(rw) * (kThreadsY + 2 * rh) + k);
  }
};

// MODE: kPearson (also SSIM), kNrmse, kCosine, kAbsDiff. Bound by FP32 issue: a
// pixel's element is 6 operations that may not be merged (sum; difference, two
// products, two sums), in packed pairs of two rows, and the window leaves 1/4 load
// a pixel. 16 frames of 1024x1024, 15x15 (149 elements), normalised: 1365 us with one
// load an element and pass and a thread per two pixels, 720 now (403 at one scalar
// operation a lane and clock).
template <int MODE, int PX>
__global__ void __launch_bounds__(32 * kThreadsY)
    k_block_map(const float* __restrict__ img_all, int W, int H, const __grid_constant__ BlockRows e,
                const __grid_constant__ RefBlock rb, int metric, f2 nz, float* __restrict__ out_all,
                float* __restrict__ stds_all, unsigned* __restrict__ mm) {
  // shared: pair row r of the tile = its rows r and r + 8 side by side, for r in
  // [0, 8 + 2 rh); then the reference block, each value twice.
  extern __shared__ f2 tile[];
  const size_t plane = (size_t)W * H * blockIdx.z;
  const float* img = img_all + plane;
  float* out = out_all + plane;
  float* stds = stds_all ? stds_all + plane : nullptr;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int cols = Tile<PX>::cols(e.rw), p = Tile<PX>::p(e.rw), pitch = PX * p;
  const int pr = kThreadsY + 2 * e.rh, K = e.k;
  f2* s_ref = tile + (size_t)pitch * pr;
  {
    const int x0 = blockIdx.x * Tile<PX>::kX - e.rw, y0 = blockIdx.y * kTileY - e.rh;
    float* t = reinterpret_cast<float*>(tile);
    for (int r = ty; r < pr + kThreadsY; r += kThreadsY) {
      const int gy = y0 + r;
      const bool row_in = gy >= 0 && gy < H;
      for (int c = tx; c < cols; c += 32) {
        const int gx = x0 + c;
        const float v = row_in && gx >= 0 && gx < W ? img[(size_t)gy * W + gx] : 0.0f;
        const int o = (c % PX) * p + c / PX;
        if (r < pr) t[2 * (r * pitch + o)] = v;
        if (r >= kThreadsY) t[2 * ((r - kThreadsY) * pitch + o) + 1] = v;
      }
    }
    for (int i = threadIdx.x; i < K; i += 32 * kThreadsY) s_ref[i] = pack2(rb.px[i], rb.px[i]);
  }
  __syncthreads();
  const int x = blockIdx.x * Tile<PX>::kX + PX * tx, y = blockIdx.y * kTileY + ty;
  unsigned lo = 0xffffffffu, hi = 0u;
  // (a pixel outside the interior is evaluated on the zero-padded tile and discarded)
  const bool some = x < W - e.rw && x + PX > e.rw && y < H - e.rh && y + kThreadsY >= e.rh;
  float val[PX][2], sd[PX][2];
#pragma unroll
  for (int q = 0; q < PX; q++) val[q][0] = val[q][1] = sd[q][0] = sd[q][1] = 0.0f;
  if (some) {
    const f2* base = tile + ty * pitch + tx;
    f2 m[PX], v[PX], a[PX], xx[PX], rr = 0;
#pragma unroll
    for (int q = 0; q < PX; q++) m[q] = v[q] = a[q] = xx[q] = 0;
    sweep<PX>(base, p, pitch, e, [&](int, auto w) {
#pragma unroll
      for (int q = 0; q < PX; q++) m[q] = add2(m[q], w(q));
    });
#pragma unroll
    for (int q = 0; q < PX; q++) {
      float s0, s1;
      unpack2(m[q], &s0, &s1);
      m[q] = pack2(__fdiv_rn(s0, (float)K), __fdiv_rn(s1, (float)K));
    }
    sweep<PX>(base, p, pitch, e, [&](int i, auto w) {
      const f2 ref = MODE == kAbsDiff ? 0 : s_ref[i];
#pragma unroll
      for (int q = 0; q < PX; q++) {
        const f2 d = sub2(w(q), m[q]);
        v[q] = add2(v[q], mul2(d, d, nz));
        if (MODE == kNrmse) {
          const f2 t = sub2(ref, d);
          a[q] = add2(a[q], mul2(t, t, nz));
        } else if (MODE == kCosine) {
          a[q] = add2(a[q], mul2(ref, w(q), nz));
          xx[q] = add2(xx[q], mul2(w(q), w(q), nz));
        } else if (MODE == kPearson) {
          a[q] = add2(a[q], mul2(ref, d, nz));
        }
      }
      if (MODE == kCosine) rr = add2(rr, mul2(ref, ref, nz));
    });
    float r0, r1;
    unpack2(rr, &r0, &r1);
#pragma unroll
    for (int q = 0; q < PX; q++) {
      float ms[2], vs[2], as[2], xs[2];
      unpack2(m[q], &ms[0], &ms[1]);
      unpack2(v[q], &vs[0], &vs[1]);
      unpack2(a[q], &as[0], &as[1]);
      unpack2(xx[q], &xs[0], &xs[1]);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float s;
        const float o = block_metric_value(metric, K, ms[h], vs[h], as[h], r0, xs[h], rb.mean, rb.std, &s);
        const int px = x + q, py = y + h * kThreadsY;
        if (px >= e.rw && px < W - e.rw && py >= e.rh && py < H - e.rh) {
          val[q][h] = o;
          sd[q][h] = s;
          lo = min(lo, ord_bits(o));
          hi = max(hi, ord_bits(o));
        }
      }
    }
  }
  const bool wide = PX == 4 && (W & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(stds) & 15) == 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int py = y + h * kThreadsY;
    if (x >= W || py >= H) continue;
    const size_t o = (size_t)py * W + x;
    if (PX == 4 && wide) {
      *reinterpret_cast<float4*>(out + o) = make_float4(val[0][h], val[1 % PX][h], val[2 % PX][h], val[3 % PX][h]);
      if (stds)
        *reinterpret_cast<float4*>(stds + o) = make_float4(sd[0][h], sd[1 % PX][h], sd[2 % PX][h], sd[3 % PX][h]);
    } else {
#pragma unroll
      for (int q = 0; q < PX; q++)
        if (x + q < W) {
          out[o + q] = val[q][h];
          if (stds) stds[o + q] = sd[q][h];
        }
    }
  }
  if (mm) cta_minmax(lo, hi, mm + 2 * blockIdx.z);
}

// Shared memory of a tile at most: the tallest block's (3x509) takes 140 KB of it.
constexpr size_t kMaxTile = 144 * 1024;
// Of the four-column tile: two CTAs an SM.
constexpr size_t kMaxTile4 = 113 * 1024;

template <int MODE, int PX>
cudaError_t launch_mode(const float* img, int w, int h, int frames, const BlockRows& e, const RefBlock& rb, int metric,
                        float* out, float* stds, unsigned* mm, cudaStream_t st) {
  const size_t smem = Tile<PX>::smem(e.rw, e.rh, e.k);
  if (smem > kMaxTile) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {  // (the same value in every call: another thread's launch may lie between)
    const cudaError_t err =
        cudaFuncSetAttribute(k_block_map<MODE, PX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxTile);
    if (err != cudaSuccess) return err;
  }
  const dim3 grid((w + Tile<PX>::kX - 1) / Tile<PX>::kX, (h + kTileY - 1) / kTileY, frames);
  k_block_map<MODE, PX><<<grid, 32 * kThreadsY, smem, st>>>(img, w, h, e, rb, metric, kNegZero2, out, stds, mm);
  return cudaGetLastError();
}

template <int PX>
cudaError_t launch_px(const float* img, int w, int h, int frames, const BlockRows& e, const RefBlock& rb, int metric,
                      float* out, float* stds, unsigned* mm, cudaStream_t st) {
  switch (metric) {
    case kNrmse: return launch_mode<kNrmse, PX>(img, w, h, frames, e, rb, metric, out, stds, mm, st);
    case kCosine: return launch_mode<kCosine, PX>(img, w, h, frames, e, rb, metric, out, stds, mm, st);
    case kAbsDiff: return launch_mode<kAbsDiff, PX>(img, w, h, frames, e, rb, metric, out, stds, mm, st);
    default: return launch_mode<kPearson, PX>(img, w, h, frames, e, rb, metric, out, stds, mm, st);
  }
}

}  // namespace

cudaError_t launch_block_map(const float* img, int w, int h, int frames, const Ellipse& e, const RefBlock& rb,
                             int metric, float* out, float* stds, unsigned* mm, int num_sms, cudaStream_t st) {
  BlockRows rows;
  rows.k = e.k;
  rows.rw = e.rw;
  rows.rh = e.rh;
  for (int i = 0; i < e.k; i++) rows.hw[e.dy[i] + e.rh] = e.dx[i];  // the last column of a row stays
  rows.single = 0;
  while (rows.single < e.rh && rows.hw[rows.single] == 0) rows.single++;
  // Four pixel columns a thread where that still gives 1.5 CTAs an SM, the
  // 128-column tiles pad the width to no more than 1.5 times what 32-column tiles do, and
  // two tiles fit an SM; else one. At 1024x1024 15x15 four take 80 us where one takes 94
  // (700x700: 55 and 61), at 400x300 15x15 (76 CTAs against 247) 44 and 40, at 513x512 9x9
  // 40 and 37; of tall blocks at 1024x1024, 5x61 (two tiles an SM) 119 and 131 and 3x81 (two) 88
  // and 85, 3x101 (one) 121 and 97, 5x101 (one) 210 and 180, and from 3x195 on the tile fits no SM.
  const int tiles = (w + Tile<4>::kX - 1) / Tile<4>::kX, ys = (h + kTileY - 1) / kTileY;
  const bool four = (long long)tiles * ys * frames * 2 >= 3LL * num_sms &&
                    2 * tiles * Tile<4>::kX <= 3 * ((w + 31) / 32 * 32) &&
                    Tile<4>::smem(e.rw, e.rh, e.k) <= kMaxTile4;
  if (four) return launch_px<4>(img, w, h, frames, rows, rb, metric, out, stds, mm, st);
  return launch_px<1>(img, w, h, frames, rows, rb, metric, out, stds, mm, st);
}

__global__ void k_init_minmax(unsigned* mm, int planes) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < planes; i += gridDim.x * blockDim.x) {
    mm[2 * i] = 0xffffffffu;
    mm[2 * i + 1] = 0u;
  }
}

namespace {

struct PlaneArgs {
  float* a;
  const float* mask;  // null: the whole interior
  int W, H, rw, rh;
  const unsigned* mm_in;
  unsigned* mm_out;  // the range of the results, or null
  int own;           // 1: a range per plane, 0: one for all (the slices of a volume)
};

// One pass over the interior (where mask > 0): see PlanePass. VEC floats a load;
// the thread's column and row advance with its index, without divisions.
template <int OP, int VEC>
__global__ void __launch_bounds__(256) k_plane_pass(const PlaneArgs g) {
  const size_t n = (size_t)g.W * g.H, step = (size_t)gridDim.x * 256 * VEC;
  float* a = g.a + n * blockIdx.y;
  const float* mask = g.mask ? g.mask + n * blockIdx.y : nullptr;
  float mn = 0.0f, d = 1.0f;
  bool remap = false;
  if (OP == kPassRemap || OP == kPassRemapInvert || OP == kPassAbsDiff) {
    const unsigned k0 = g.mm_in[2 * g.own * blockIdx.y], k1 = g.mm_in[2 * g.own * blockIdx.y + 1];
    remap = k1 != 0u || OP == kPassAbsDiff;  // nothing selected: the reference remaps nothing either
    mn = ord_float(k0);
    float mx = ord_float(k1);
    if (OP == kPassAbsDiff) mx = fmaxf(mx, 1.4e-45f);
    d = __fadd_rn(__fsub_rn(mx, mn), kEps);
  }
  size_t p = ((size_t)blockIdx.x * 256 + threadIdx.x) * VEC;
  int x = (int)(p % g.W), y = (int)(p / g.W);
  const int sx = (int)(step % g.W), sy = (int)(step / g.W);
  unsigned lo = 0xffffffffu, hi = 0u;
  for (; p < n; p += step) {
    float v[VEC], m[VEC];
    if (VEC == 4) {
      const float4 t = *reinterpret_cast<const float4*>(a + p);
      v[0] = t.x, v[1 % VEC] = t.y, v[2 % VEC] = t.z, v[3 % VEC] = t.w;
      if (mask) {
        const float4 u = *reinterpret_cast<const float4*>(mask + p);
        m[0] = u.x, m[1 % VEC] = u.y, m[2 % VEC] = u.z, m[3 % VEC] = u.w;
      }
    } else {
      v[0] = a[p];
      if (mask) m[0] = mask[p];
    }
    int xx = x, yy = y;
    bool any = false;
#pragma unroll
    for (int q = 0; q < VEC; q++) {
      const bool in = xx >= g.rw && xx < g.W - g.rw && yy >= g.rh && yy < g.H - g.rh;
      if (OP == kPassMask && in) {  // (a map is 0 outside its interior)
        v[q] = __fmul_rn(v[q], m[q]);
        any = true;
      }
      if (in && (!mask || m[q] > 0.0f)) {
        if (remap) v[q] = __fdiv_rn(__fsub_rn(v[q], mn), d);
        if (OP == kPassAbsDiff) v[q] = __fsub_rn(1.0f, v[q]);
        if (OP == kPassRemapInvert) v[q] = (v[q] == 0.0f) ? 1.0f : __fdiv_rn(1.0f, v[q]);
        lo = min(lo, ord_bits(v[q]));
        hi = max(hi, ord_bits(v[q]));
        any = true;
      }
      if (++xx == g.W) xx = 0, yy++;
    }
    if (OP != kPassRange && any) {
      if (VEC == 4) *reinterpret_cast<float4*>(a + p) = make_float4(v[0], v[1 % VEC], v[2 % VEC], v[3 % VEC]);
      else a[p] = v[0];
    }
    x += sx;
    y += sy;
    if (x >= g.W) x -= g.W, y++;
  }
  if (g.mm_out) cta_minmax(lo, hi, g.mm_out + 2 * g.own * blockIdx.y);
}

template <int VEC>
void launch_pass(PlanePass op, const PlaneArgs& g, dim3 grid, cudaStream_t st) {
  switch (op) {
    case kPassRange: k_plane_pass<kPassRange, VEC><<<grid, 256, 0, st>>>(g); break;
    case kPassRemap: k_plane_pass<kPassRemap, VEC><<<grid, 256, 0, st>>>(g); break;
    case kPassRemapInvert: k_plane_pass<kPassRemapInvert, VEC><<<grid, 256, 0, st>>>(g); break;
    case kPassMask: k_plane_pass<kPassMask, VEC><<<grid, 256, 0, st>>>(g); break;
    case kPassAbsDiff: k_plane_pass<kPassAbsDiff, VEC><<<grid, 256, 0, st>>>(g); break;
  }
}

}  // namespace

void launch_plane_pass(PlanePass op, float* a, const float* mask, int w, int h, int rw, int rh, int planes,
                       const unsigned* mm_in, unsigned* mm_out, int num_sms, cudaStream_t st, bool shared_range) {
  if (planes < 1) return;
  const PlaneArgs g{a, mask, w, h, rw, rh, mm_in, mm_out, shared_range ? 0 : 1};
  const size_t n = (size_t)w * h;
  // float4 where every plane and quad is aligned
  const bool vec = n % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(mask)) & 15) == 0;
  const size_t per = 256 * (vec ? 4 : 1), want = (n + per - 1) / per;
  const size_t cap = std::max<size_t>(1, (size_t)16 * num_sms / planes);
  const dim3 grid((unsigned)std::min(want, cap), planes);
  if (vec) launch_pass<4>(op, g, grid, st);
  else launch_pass<1>(op, g, grid, st);
}

}  // namespace sred
