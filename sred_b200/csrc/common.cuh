// Shared definitions of libsred's device code and host orchestration.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/sred.h"

namespace sred {

constexpr float kEps = 0.0000001f;  // java/Utils.java:20 (Utils.EPSILON)
constexpr float kC1 = 0.0001f;      // cl/kernelGetGlobalSsim2D.cl:102
constexpr float kC2 = 0.0009f;      // cl/kernelGetGlobalSsim2D.cl:104
constexpr int kMaxK = 512;          // largest ellipse block size accepted
constexpr int kMaxGlobalK = 212;    // largest block of a global map
constexpr size_t kMaxSmem = 227 * 1024;  // shared memory of a CTA

enum Metric { kPearson = 0, kSsim = 1, kNrmse = 2, kAbsDiff = 3, kCosine = 4,
              kDebugDot = 5 /* diagnostics: num += G a_p a_q */,
              kHu = 6, kPhase = 7 /* block-map shape metrics */,
              kNrmseW = 8 /* NRMSE with each term weighted (the 3D global kernel) */,
              // NRMSE from the accumulated squared difference of the unit
              // vectors (FP32 engine): unweighted (2D) and weighted (3D)
              kNrmseD = 9, kNrmseDW = 10,
              kHu7 = 11 /* block map: distance of the seven Hu invariants */,
              kDebugSum = 12 /* diagnostics: num += r_p + r_q */ };

// The FP32 engine's accumulator holds sum_i (u_p,i - u_q,i)^2 instead of the
// dot product for these metrics.
__host__ __device__ constexpr bool diff_metric(int m) { return m == kNrmseD || m == kNrmseDW; }

// Ellipse pixel offsets (dx, dy), row-major ellipse order, as the kernels gather them.
struct Ellipse {
  int k;
  int rw, rh;
  short dx[kMaxK];
  short dy[kMaxK];
};

// Host: build the ellipse (java/GlobalRepetition2D_.java:102-111).
int build_ellipse(int bw, int bh, Ellipse* e);

// ---------------------------------------------------------------------------
// Per-block data of the global map, produced by the moment pass.
//   gram list: relevant, non-flat blocks (enter the all-pairs contraction)
//   flat list: relevant blocks with sigma == 0 (handled in closed form)
// ---------------------------------------------------------------------------
struct BlockParams {
  float a;      // sigma64 * sqrt(log2(e) / (noise_var + eps)): weight = 2^-(a_p - a_q)^2
  float e;      // eps / sigma64 (0 if sigma64 == 0)
  float r;      // 1 / sigma64 (0 if sigma64 == 0)
  float sigma;  // sigma64
  float mu;     // mu64
  float pad0, pad1, pad2;
};

// Split-FP16 operand of the tensor-core engine: u = hi + mid (+ lo), hi = fp16(u 2^14),
// mid = fp16(u 2^14 - hi), lo = fp16(u 2^14 - hi - mid) (|u| <= 1, so hi <= 2^14 and every
// mid down to u = 2^-16 keeps its 11 bits); G = 2^-28 of the accumulated value.
//   two parts:   hi.hi + hi.mid + mid.hi; an element is off by up to 2^-23 of its binade and the
//                product by mid.mid (2^-22 at most)
//   three parts: hi.hi + hi.mid + mid.hi + mid.mid + hi.lo + lo.hi: FP32-level elements. While
//                6 K <= 128, where a tile's time is its epilogue's (split_parts).
//
// A row holds each part once. The row and the column operand are the same array:
// the MMAs pair blocks of 16 elements of one with blocks of the other. K = 16 nb + r:
//   [hi: nb blocks | mid: nb blocks | lo: nb blocks | row tail: nt | column tail: nt],
// the tails holding the last r elements of every part side by side, as
// [mid|hi|hi] in the row tail and [hi|mid|hi] in the column tail ([lo|mid|hi|mid|hi|hi] and
// [hi|mid|lo|hi|mid|hi] of three parts: smallest products first), nt blocks: 3 nb + nt steps
// of 16 instead of 3 ceil(K / 16) (6 nb + nt of 6 ceil(K / 16)).
struct SplitLayout {
  int parts, nb, r, nt, pitch;  // pitch: fp16 per row, a multiple of 32
  __host__ __device__ int steps() const { return parts * (parts + 1) / 2 * nb + nt; }
};
__host__ __device__ inline int split_parts(int K) { return 6 * K <= 128 ? 3 : 2; }
__host__ __device__ inline SplitLayout split_layout(int K) {
  const int parts = split_parts(K);
  int nb = K / 16, r = K % 16;
  if (parts == 3 && r > 5) nb++, r = 0;  // (a padded block: fewer columns than a tail of six r)
  const int nt = (parts * (parts + 1) / 2 * r + 15) / 16;
  return SplitLayout{parts, nb, r, nt, (16 * (parts * nb + 2 * nt) + 31) / 32 * 32};
}
constexpr float kSplitScale = 16384.0f;
constexpr float kSplitGScale = 1.0f / (16384.0f * 16384.0f);
constexpr int kSplitSlack = 32;  // fp16 past the last row that a copy may read
// K': the padded contraction length (the key of the launch-shape table).
inline int split_cols(int K) { return (3 * K + 31) / 32 * 32; }
inline bool nrmse_metric(int m) { return m == 2 /* kNrmse */ || m == 8 /* kNrmseW */; }

// Element i of a block's vector (already scaled) into its row.
__device__ __forceinline__ void store_split(__half* row, const SplitLayout& l, int i, double u) {
  const __half hi = __float2half_rn((float)u);
  const double rest = u - (double)__half2float(hi);
  const __half mid = __float2half_rn((float)rest);
  const int n = 16 * l.nb, r = l.r;
  __half* a = row + l.parts * n + (i - n);  // (i in the tail)
  __half* b = a + 16 * l.nt;
  if (l.parts == 2) {
    if (i < n) {
      row[i] = hi;
      row[n + i] = mid;
    } else {
      a[0] = mid, a[r] = hi, a[2 * r] = hi;
      b[0] = hi, b[r] = mid, b[2 * r] = hi;
    }
    return;
  }
  const __half lo = __float2half_rn((float)(rest - (double)__half2float(mid)));
  if (i < n) {
    row[i] = hi;
    row[n + i] = mid;
    row[2 * n + i] = lo;
  } else {
    a[0] = lo, a[r] = mid, a[2 * r] = hi, a[3 * r] = mid, a[4 * r] = hi, a[5 * r] = hi;
    b[0] = hi, b[r] = mid, b[2 * r] = lo, b[3 * r] = hi, b[4 * r] = mid, b[5 * r] = hi;
  }
}
// The zeros behind the tails and behind the last block's elements, one of 32 lanes' share.
__device__ __forceinline__ void store_split_pad(__half* row, const SplitLayout& l, int K, int lane) {
  const __half zero = __float2half_rn(0.0f);
  __half* tail = row + 16 * l.parts * l.nb;
  for (int i = l.parts * (l.parts + 1) / 2 * l.r + lane; i < 16 * l.nt; i += 32) tail[i] = tail[16 * l.nt + i] = zero;
  if (l.parts == 3)  // (two parts pad no block)
    for (int i = K + lane; i < 16 * l.nb; i += 32)
      for (int p = 0; p < 3; p++) row[16 * l.nb * p + i] = zero;
}

// a / b, correctly rounded, for many a and one b: y = RN(1/b) once, then
// q = RN(a y), the exact residual r = a - b q (one FMA) and RN(q + r y).
// Markstein's theorem (P. Markstein, IBM J. Res. Dev. 34(1):111-119, 1990)
// makes the result the correctly rounded quotient when y is the correctly
// rounded reciprocal and q is within one ulp, barring underflow; tested
// against IEEE division (sred_debug_divide_fixed).
__device__ __forceinline__ float div_fixed(float a, float b, float y) {
  const float q = __fmul_rn(a, y);
  const float r = __fmaf_rn(-q, b, a);
  return __fmaf_rn(r, y, q);
}
// The same in FP64 (y = RN(1/b) from __drcp_rn); tested against IEEE
// division (sred_debug_divide_fixed64).
__device__ __forceinline__ double div_fixed(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  const double r = __fma_rn(-q, b, a);
  return __fma_rn(r, y, q);
}

// Epilogue constants shared by all tiles of one map.
struct EpiConsts {
  int metric;
  int n;            // valid blocks (rows == cols)
  float nrmse_scale;  // (K-1)/K
  float c1, c2;
  // NRMSE on the tensor cores: pairs with G above nrmse_near get the term of
  // the exact squared difference of their FP32 unit vectors U (row pitch kp,
  // K values), the form the FP32 engine evaluates for every pair.
  const float* U = nullptr;
  int kp = 0, K = 0;
  float nrmse_near = 1.0f;
  float gscale = 1.0f;      // G = gscale x the contraction's accumulator
  float inv_wscale = 0.0f;  // sigma / a
  float tau = 0.0f;         // eps (a / sigma)^2: Pearson's t = tau / (a_p a_q)
  float c2h = 0.0f;         // c2 / (2 gscale)
};

// Near-identical pairs (G > 1 - 2^-7) of tensor-core NRMSE take the exact
// difference form: there 1 - G is within an order of magnitude of the FP32
// accumulation error of G, which the square root of the term amplifies.
constexpr float kNrmseNear = 1.0f - 1.0f / 128.0f;

// Launch the FP32 CUDA-core all-pairs kernel (global_fp32.cu), on the same
// symmetric schedule as the tensor-core engine with 128 x 128 tiles.
// U: n_pad x kp floats (unit vectors), params: n_pad entries, num: n
// doubles (zeroed). The work items are split into n_shards equal ranges; this
// launch runs range `shard`. arange (Abs-diff): the range of a, by which the
// kernel leaves the sums to launch_absdiff.
cudaError_t launch_gram_fp32(const float* U, int kp, const BlockParams* params, const float* tile_rmax,
                             EpiConsts ec, double* num, int num_sms, cudaStream_t st, int shard = 0,
                             int n_shards = 1, const unsigned* arange = nullptr);

// Column parameters of one BN-column tile as the tensor-core engine copies
// them into shared memory: [a x BN | r x BN | sigma x BN | mu x BN | per group
// of BN/4 columns {centre of a, half range of a, centre of r, half range of r}],
// each array permuted within every 16-column group so that an epilogue thread's
// four columns of the group (2j, 2j + 1, 8 + 2j, 9 + 2j for j = t % 4) are one
// float4.
__host__ __device__ constexpr int col_soa_floats(int bn) { return 4 * bn + 16; }
__host__ __device__ constexpr int col_soa_pos(int i) {
  return (i & ~15) + 4 * ((i & 7) >> 1) + 2 * ((i >> 3) & 1) + (i & 1);
}
// Row parameters of one 128-row block: [a | r | sigma | mu] x 128, then the same
// four values per group of 32 rows.
constexpr int kRowSoaFloats = 4 * 128 + 16;

// Ring shape of the tensor-core engine for K ellipse pixels: stages of whole
// row-block tiles or of single 64-column chunks (sc chunks each), dynamic shared
// memory. False if the operands do not fit in shared memory (K = 267-271, 278-287, above 288).
struct TcPlan {
  int ctas;  // CTAs that share a tile (1 or 2)
  int sc, stages;
  size_t smem;
};
bool plan_gram_tc(int K, TcPlan* plan);

// What a status word of the tensor-core kernel other than 0 means (kTcUnaligned: shared memory
// not on the 1,024-byte boundary the swizzled tiles need; the others: the role whose wait ran out).
constexpr int kTcUnaligned = 5;
inline sred_status tc_status_error(int status, const char** msg) {
  if (status == kTcUnaligned) {
    *msg = "tensor-core kernel: shared memory not aligned to 1,024 bytes";
    return SRED_ERR_LAUNCH;
  }
  *msg = "tensor-core pipeline wait exceeded its bound";
  return SRED_ERR_TIMEOUT;
}

// Test hooks of the tensor-core engine: a wait limit (0: 4 s) and a tile whose
// operand copies the producer never issues (-1: none), so that the pipeline
// waits run out with nothing in flight.
struct TcDebug {
  unsigned long long timeout_ns;
  long long withhold_tile;
};

// A launch shape of the tensor-core engine (bn 0: the default plan): tr 1 for
// whole-tile stages, 0 for single chunks; L: the largest run of row blocks per
// work item (the item-count rule may lower it). The tiles are 256 columns wide;
// 128, a width of earlier tables, runs as 256.
struct TcChoice {
  int bn = 0, tr = 0, L = 0;
};
// The launch shapes to time for K (at most cap), and whether one can run.
int gram_tc_candidates(int K, TcChoice* out, int cap);
bool gram_tc_valid(int K, const TcChoice& c);

// Floats of the parameter workspace launch_gram_tc fills (column tiles and
// row blocks) for n_pad blocks.
size_t gram_tc_soa_floats(int n_pad);

// Work items of the symmetric schedule for n blocks and tile width bn (the
// upper triangle of 128-row x bn-column tiles in runs of L row blocks).
long long gram_tc_items(int n, int bn, int* L, int num_sms, int max_L = 0);

// Launch the split-FP16 tcgen05 all-pairs kernel (global_tc.cu).
// U: n_pad rows of split_layout(K).pitch fp16 (store_split; rows past n zero);
// params: n_pad entries (rows past n zero); soa_ws: gram_tc_soa_floats(n_pad)
// floats of workspace; num: n doubles (zeroed), to which every pair's term is
// added for both blocks. The upper-triangle work items are split into n_shards
// equal ranges; this launch runs range `shard` (the shards' num add up to the
// whole map).
cudaError_t launch_gram_tc(const __half* U, int K, int n_pad, const BlockParams* params, float* soa_ws, EpiConsts ec,
                           double* num, int num_sms, int* status, cudaStream_t st, int shard = 0, int n_shards = 1,
                           const TcDebug* dbg = nullptr, const TcChoice* choice = nullptr);

}  // namespace sred
