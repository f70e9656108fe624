// Split-FP16 tcgen05 engine of the global repetition map (sm_100a).
//
// G = <u_p, u_q> on the 5th-generation tensor cores, where each block's FP64 unit
// vector u is split into fp16 parts, u = hi + mid, and lo for small blocks (common.cuh:
// SplitLayout), and G = hi.hi + mid.hi + hi.mid (+ mid.mid + lo.hi + hi.lo) with FP32
// accumulation: what two parts leave out is below 3 2^-22 |u_p| |u_q| (mid.mid, and the
// rounding of each mid).
//
// Symmetric schedule. Every per-pair term of the global map (weight, Pearson,
// global SSIM, NRMSE; epilogue.cuh) is symmetric in (p, q), so each unordered
// pair is evaluated once: only tiles of the upper triangle are scheduled (a
// 128-row block rb against a 256-column tile ct with 128 rb <= 256 ct + 255), pairs
// below the diagonal are masked in the diagonal tiles, and each pair's term is
// added to the sums of both blocks (the self pair once).
//
// Work item = (column tile ct, a run of up to L row blocks). The column tile's operand
// stays in shared memory for the whole item, the row blocks stream through a ring of
// stages. Where the operand and three whole row-block tiles fit one CTA (K up to 42,
// and 48-53, 64), a CTA works on an item by itself with M = 128 MMAs. Else a cluster of
// two CTAs (two SMs) does: row blocks go in pairs, CTA r of the cluster takes row block
// rb + r, one M = 256 tcgen05.mma (cta_group::2) computes both CTAs' 128 x 256 tiles,
// and each CTA keeps half of the column tile's operand (128 rows of U), with whole row
// blocks as stages or, from K = 97 on (and for some from 75), chunks of 64 columns. One
// CTA per tile reads 96 bytes of shared memory per clock for the MMAs alone, of 128 there
// are, and writes 32 more for the row blocks; the pair reads 64. Items are ordered panel-major
// (decode_item): all clusters work on the same row blocks at a time and share them
// in L2, and a panel's column tiles stay in L2 while the runs pass over them.
// Each cluster (or CTA) walks its items twice: first their full tiles, then their masked
// ones (diagonal and ragged tiles, about 0.2% of all), so that the masked
// epilogue form sits in a loop of its own (with it in the main loop the full
// tiles ran 3% slower).
// Warp roles (one CTA per SM, persistent):
//   warp 0      TMA producer (one thread)
//   warp 1      CTA 0: MMA issuer (one thread): tcgen05.mma M=128 or 256, N=256, K=16
//               into one of two TMEM accumulators, tcgen05.commit to both CTAs'
//               barriers. CTA 1: relays its producer's arrivals to CTA 0.
//   warps 2-17  epilogue: tcgen05.ld.16x256b gives each thread 4 rows x 4 columns
//               of a 32 x 16 block; the fused per-pair metric runs on f32x2 pairs
//               of neighbouring columns. Column sums of the item stay in registers
//               and leave once per item (a butterfly over the 8 lanes that share
//               columns); row sums leave once per tile (a butterfly over 4 lanes):
//               one FP64 atomic add per row and warp.
// Every mbarrier wait is bounded by wall time (a host-set limit); on expiry the
// kernel records a status code, stops issuing work, waits (bounded) for its own
// copies in flight, frees TMEM and returns. No TMA multicast is used.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "epilogue.cuh"

namespace sred {

namespace {

constexpr int kBM = 128;                          // rows per CTA and tile (TMEM lanes)
constexpr int kBN = 256;                          // columns per tile
constexpr int kChunk = 64;                        // fp16 per chunk (128 B: one SWIZZLE_128B atom row)
constexpr int kChunkBytes = kBM * kChunk * 2;     // 128 rows of a chunk: 16 KB
constexpr int kMaxStages = 16;
constexpr int kEpiWarps = 16;                     // 4 per SM sub-partition
constexpr int kThreads = (kEpiWarps + 2) * 32;
constexpr int kRSlots = 4;                        // row-parameter ring depth
constexpr int kRowR = kBM, kRowS = 2 * kBM, kRowMu = 3 * kBM;  // r, sigma, mu of a row block (a at 0)
constexpr int kRowGrp = 4 * kBM;                  // the four 32-row groups' centres and half ranges
constexpr int kRowFloats = kRowSoaFloats;         // one 128-row block's parameters
constexpr int kColFloats = col_soa_floats(kBN);   // one column tile's parameters
constexpr int kMaxRun = 128;                      // row blocks per run (work item), at most
constexpr int kBarBytes = 512;
constexpr int kMaxMma = 64;                       // entries of the MMA table (SplitLayout::steps() + 1 at most 58)
constexpr int kTabBytes = kMaxMma * 8 + 16 * 4;

enum { ST_OK = 0, ST_TIMEOUT_PRODUCER = 1, ST_TIMEOUT_MMA = 2, ST_TIMEOUT_EPI = 3, ST_TIMEOUT_DRAIN = 4, ST_ALIGNMENT = kTcUnaligned };

// Epilogue sets. Two: warps 0-7 take the even tiles, warps 8-15 the odd ones, each
// warp 32 rows x 128 columns, so that one set's fixed work per tile (waits, row
// and column factors, row sums) is spread over more pairs and runs under the
// other set's pair loop. One: all 16 warps share every tile, 32 x 64 each, which
// halves the column sums a thread holds and leaves registers for the row
// constants of SSIM and NRMSE (96 per thread).
template <int METRIC>
constexpr int epi_sets() {
  return METRIC == kPearson ? 2 : 1;
}
template <int METRIC>
struct Cfg {
  static constexpr int kSets = epi_sets<METRIC>();
  static constexpr int kColW = 64 * kSets;          // columns per epilogue warp (a slab)
  static constexpr int kCH = kColW / 16;            // 16-column chunks per slab
};
constexpr int kScratch = 32 + 128;                  // floats of f and g per epilogue warp

struct TcArgs {
  int parts, nb, nt;            // parts, blocks of 16 per part and tail blocks (SplitLayout)
  int nch, sc, nst, stages;     // chunks per tile, chunks per stage, stages per tile, ring depth
  int n_rb, n_ct;               // row blocks holding valid rows, column tiles
  int L, h;                     // row blocks per item (a run), L / (BN / 128)
  int n_runs;                   // runs of L row blocks
  int panel, n_panels;          // column tiles per panel (panel-major item order), panels
  long long item0, item1;       // items of this launch
  const float* colsoa;          // per column tile, permuted (col_soa_pos)
  const float* rowsoa;          // per 128-row block, natural order
  EpiConsts ec;
  double* num;
  int* status;
  unsigned long long timeout_ns;
  long long withhold;           // test hook: the producers never issue this tile's loads (-1: none)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Address of the same shared-memory location in CTA 0 of the cluster.
__device__ __forceinline__ uint32_t leader_addr(uint32_t a) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(a));
  return r;
}

// Arrive on a barrier of either CTA of the cluster (a shared::cluster address).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// The epilogue's arrivals hand a buffer that this warp has read to the copies or MMAs that
// overwrite it.
// The accumulator's: tensor memory, whose reads tcgen05.wait::ld completes and
// tcgen05.fence::before_thread_sync orders before the arrival, so that one is relaxed (a release
// at cluster scope cost 1,500 clocks a tile).
__device__ __forceinline__ void mbar_arrive_tmem(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The shared-memory buffers' (barriers of this CTA): one fence orders the warp's reads before
// them, the lanes' by the __syncwarp that precedes it. It waits for the warp's row-sum
// atomics in flight to reach L2 too, so it stands before a tile's, when the previous tile's
// are long there: behind them it cost 550 clocks a tile.
__device__ __forceinline__ void fence_reads() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_fenced(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase with the given parity. Returns false (and
// records `code`) if the wait exceeded the limit or another role of any CTA
// already gave up. Drain waits (for copies or MMAs this CTA issued) pass
// abort = false: they keep waiting, within the same bound, after another
// role has given up. The producer, which runs buffers ahead, backs off with a
// short nanosleep so that its polling does not take issue slots from the
// epilogue warps of its SM sub-partition; the MMA issuer does not (a late wake
// is idle tensor time: with a back-off of up to 0.5 us for both roles the 9x9
// map's MMAs waited for operands that had landed).
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, int* status, unsigned long long limit_ns,
                                            int code, bool abort, bool backoff) {
  const unsigned long long t0 = globaltimer();
  for (uint32_t i = 1;; i++) {
    if (backoff) __nanosleep(40);
    if (mbar_test(bar, parity)) return true;
    if ((i & (backoff ? 63u : 255u)) == 0) {
      if (abort && *reinterpret_cast<volatile int*>(status) != ST_OK) return false;
      if (globaltimer() - t0 > limit_ns) {
        atomicCAS(status, ST_OK, code);
        return false;
      }
    }
  }
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const TcArgs& g, int code, bool abort = true,
                                          bool backoff = false) {
  return mbar_test(bar, parity) || mbar_wait_slow(bar, parity, g.status, g.timeout_ns, code, abort, backoff);
}

// The same for a whole warp, with one answer for all its lanes.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, const TcArgs& g, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, g, code));
}
// One box of U: g.sc chunks of 64 columns of 128 rows (a stage, or the whole half
// of a column tile), from chunk c and row y. One instruction per operand tile: the
// producer thread needs some 150 clocks for each, and seven a tile (one per chunk,
// one L2 prefetch per chunk, the row parameters) bounded the pipeline at 1,700.
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int y, int c) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(y), "r"(c)
      : "memory");
}

// L2 prefetch of one box (no shared memory, no completion).
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int y, int c) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(0), "r"(y), "r"(c)
               : "memory");
}

// Plain bulk copy (no tensor map): 16-byte aligned addresses, size a multiple of 16.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}

// Shared-memory matrix descriptors: K-major, SWIZZLE_128B (128-byte rows), 8-row
// groups 1,024 B apart. Only the start address (16-byte units, low word) differs
// between operands; the rest is the constant high word (stride 64 units,
// descriptor version 1, swizzle mode 2).
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }

// Instruction descriptor, kind::f16: D = F32, A = B = FP16, both K-major, M = 128
// rows per CTA of the group, N = 256.
template <int CTAS>
constexpr uint32_t idesc() {
  return (1u << 4) | (static_cast<uint32_t>(kBN >> 3) << 17) | (static_cast<uint32_t>(CTAS * kBM >> 4) << 24);
}

template <int CTAS>
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint32_t da_lo, uint32_t db_lo, uint32_t accumulate) {
  if constexpr (CTAS == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %3};\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}" ::"r"(tmem_d),
        "r"(da_lo), "r"(db_lo), "n"(kDescHi), "n"(idesc<2>()), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %3};\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}" ::"r"(tmem_d),
        "r"(da_lo), "r"(db_lo), "n"(kDescHi), "n"(idesc<1>()), "r"(accumulate)
        : "memory");
}

// Arrive on this barrier (in both CTAs of a pair) once every MMA issued so far is complete.
template <int CTAS>
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  if constexpr (CTAS == 2)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((unsigned short)3)
        : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Issue a load of 16 lanes x 16 columns of 32-bit accumulator (no wait).
// Thread t receives lanes t/4 and t/4 + 8, columns 2(t%4), 2(t%4) + 1 of
// each 8-column half: v[0..1] (lane t/4, cols 0-7), v[2..3] (lane t/4 + 8),
// v[4..5] and v[6..7] the same for columns 8-15.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

// A batch: 16 columns of all 32 lanes.
__device__ __forceinline__ void tmem_ld_batch(uint32_t taddr, uint32_t (&v)[2][8]) {
  tmem_ld8(taddr, v[0]);
  tmem_ld8(taddr + (16u << 16), v[1]);
}

// Wait for every TMEM load this thread issued; the register operands tie
// later uses of v to the wait, so none is scheduled before it.
__device__ __forceinline__ void tmem_wait8(uint32_t (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
               :);
}
__device__ __forceinline__ void tmem_wait_batch(uint32_t (&v)[2][8]) {
  tmem_wait8(v[0]);
  tmem_wait8(v[1]);
}

// ---------------------------------------------------------------------------
// Epilogue arithmetic on f32x2 pairs (two neighbouring columns of one row).
//
// The blocks are ordered by sigma, so the 32 rows and 64 or 128 columns of a warp's
// slab have nearly equal a (the weight's argument). With a_p = alpha + dp and
// a_q = beta + dq (alpha, beta: the slab's group centres),
//   2^-(a_p - a_q)^2 = 2^-(a_p - beta)^2 * 2^(dq (2 (alpha - beta) - dq)) * 2^(2 dp dq)
//                    = f_p * g_q * 2^(2 dp dq),
// and the last factor is 1 + 2 ln2 dp dq + O((dp dq)^2). A slab whose largest
// 2 ln2 |dp dq| is below kPureTol therefore needs no exponential per pair, and
// no weight: its row sums are f_p sum_q g_q x_pq and its column sums
// g_q sum_p f_p x_pq, with f and g computed once per row and column of the
// slab (96 exponentials for 2,048 pairs). Up to kFirstTol the first-order
// factor is applied per pair. The other smooth factors of a metric (Pearson's
// 1/(1 + t), SSIM's 1/(sigma_p^2 + sigma_q^2 + c2)) split the same way; what
// the split neglects is bounded per slab, and a slab over any bound (or with a
// non-finite parameter) takes the pairwise form.
// ---------------------------------------------------------------------------

// Largest neglected relative term of a factorised weight: 2^-21 (4.8e-7, in one
// corner of a slab; it changes sign with dp and dq, so the sums are off by far
// less), the rounding error of the pairwise argument (a_p - a_q)^2 at weights
// near 2^-8. First order: (6.9e-4)^2 / 2 = 2.4e-7.
constexpr float kPureTol = 4.8e-7f;
constexpr float kFirstTol = 6.9e-4f;
// 2^-161 flushes to 0 in ex2.approx.ftz with any FP32 partner: all pair terms are 0.
constexpr float kZeroDist = 12.7f;

enum SlabMode { kZero = 0, kPure = 1, kFirst = 2, kPairFirst = 3, kPairExact = 4 };

template <int METRIC>
constexpr bool weighted_num() {
  return METRIC == kPearson || METRIC == kSsim || METRIC == kNrmseW;
}
template <int METRIC>
constexpr bool nrmse_tc() {
  return METRIC == kNrmse || METRIC == kNrmseW;
}

// What a factorised slab needs beside its parameters: the row factor is
// f_p = 2^(-(a_p - beta)^2 + sf (a_p - alpha)) cf, the column factor
// g_q = 2^(dq (eg - dq)), and kc dp dq the first-order term. Pearson's
// 1/(1 + t), t = eps / (sigma_p sigma_q) = tau / (a_p a_q), is cf = 1/(1 + t0)
// at the centres and, to first order in dp and dq, a linear term in each
// exponent (sf and part of eg).
struct SlabC {
  float alpha, beta, cf, sf, eg, kc;
};

// SSIM's 1/(sigma_p^2 + sigma_q^2 + c2): whether the mixed curvature of its logarithm,
// h = 4 x y / (x^2 + y^2 + c2)^2 at x = sigma_p and y = sigma_q, stays near its value at the
// slab's centres, which e = h ra rb holds. Over relative half ranges u and v of up to 1/16 it
// changes by at most 6 (u + v) of itself, so the first-order term neglects at most
// 6 (u + v) e: below 2^-22 here. u and v are also those of r = 1 / sigma, whose test includes
// that no sigma of the slab is 0. (The bound costs 1% of a 512x512 9x9 map.)
__host__ __device__ inline bool ssim_split_bounded(const float4& rg, const float4& cg, float e) {
  const bool ok = rg.z > 16.0f * rg.w && cg.z > 16.0f * cg.w;
  if (e <= 3e-7f) return ok;
  return ok && e * (rg.y * cg.x + cg.y * rg.x) <= 3.8e-8f * (rg.x * cg.x);
}

// Whether the row factors 2^-(a_p - beta)^2 of a slab, D between the centres, stay normal numbers.
// One that flushes to 0 takes weights of up to 2^-78 with it (g reaches 2^48); they matter to
// weighted NRMSE alone, whose self pair is 0: of a block among equal ones they are the whole sum.
__host__ __device__ inline bool row_factors_normal(float D, float ra) { return fabsf(D) + ra <= 11.2f; }

// The form a slab takes. rg, cg: {centre of a, half range of a, centre of r, half range of r}.
template <int METRIC>
__device__ __forceinline__ int slab_mode(const float4& rg, const float4& cg, const EpiConsts& ec, SlabC& sc) {
  const float D = rg.x - cg.x;
  sc.alpha = rg.x;
  sc.beta = cg.x;
  sc.cf = nrmse_tc<METRIC>() ? 1.0f : ec.gscale;  // (NRMSE scales G itself)
  sc.sf = 0.0f;
  sc.eg = 2.0f * D;
  sc.kc = 1.3862944f;  // 2 ln2
  if (fabsf(D) - rg.y - cg.y > kZeroDist) return kZero;
  bool ok = fabsf(D) * cg.y <= 24.0f;
  if (METRIC == kNrmseW) ok = ok && row_factors_normal(D, rg.y);
  if (METRIC == kPearson) {
    const float ra = rcp_approx(rg.x), rb = rcp_approx(cg.x);
    const float t0 = ec.tau * ra * rb, c = rcp_approx(1.0f + t0), u = 1.442695f * t0 * c;
    sc.cf *= c;
    sc.sf = u * ra;
    sc.eg = fmaf(u, rb, sc.eg);
    // the neglected second order of t: t0 times the squared relative ranges
    const float q = rg.y * ra + cg.y * rb;
    ok = ok && q <= 0.25f && t0 * q * q <= 1.2e-7f && t0 < 0.125f;
  }
  if (METRIC == kSsim) {
    // 1/(sigma_p^2 + sigma_q^2 + c2) splits through the centres; its mixed second
    // derivative joins the first-order term. 2 sp sq G + c2 = 2 sp sq (G + c2/2 rp rq)
    // needs sigma > 0 and no overflow.
    const float sa = rg.x * ec.inv_wscale, sb = cg.x * ec.inv_wscale;
    const float S = rcp_approx(fmaf(sa, sa, fmaf(sb, sb, ec.c2))) * ec.inv_wscale;
    const float h = 4.0f * (sa * S) * (sb * S);
    sc.kc += h;
    ok = ok && ssim_split_bounded(rg, cg, h * rg.y * cg.y) && (rg.z + rg.w) * (cg.z + cg.w) < 1e25f;
  }
  const float e = sc.kc * rg.y * cg.y;
  if (ok && e <= kFirstTol) return e <= kPureTol ? kPure : kFirst;
  if (METRIC == kPearson && kEps * (rg.z + rg.w) * (cg.z + cg.w) < kTFirst) return kPairFirst;
  return kPairExact;
}

// Row constants of the pairwise forms, both halves equal (only the fields a metric uses survive).
struct RowC {
  F2 a, ne, r;                 // weight argument, -eps/sigma, 1/sigma (diagnostic terms)
  F2 mu2, sg2, mumu, s2, sg;   // 2 mu, 2 sigma, mu^2, sigma^2 + c2, sigma
};

template <int METRIC>
__device__ __forceinline__ RowC make_rowc(const float* __restrict__ rs, int row, const EpiConsts& ec) {
  RowC c;
  auto dup = [](float v) { return f2(v, v); };
  c.a = dup(rs[row]);
  if (METRIC == kPearson) c.ne = dup(-kEps * rs[kRowR + row]);
  if (METRIC == kDebugDot || METRIC == kDebugSum) c.r = dup(rs[kRowR + row]);
  if (METRIC == kSsim || nrmse_tc<METRIC>()) {
    c.sg = dup(rs[kRowS + row]);
    c.sg2 = add2(c.sg, c.sg);
    if (METRIC == kSsim) {
      const F2 m = dup(rs[kRowMu + row]);
      c.mu2 = add2(m, m);
      c.mumu = mul2(m, m);
      c.s2 = fma2(c.sg, c.sg, f2(ec.c2, ec.c2));
    }
  }
  return c;
}

// NRMSE term of two pairs: sqrt(((K-1)/K)((s_p - s_q)^2 + 2 s_p s_q (1 - G))).
// sqrt.approx (PTX: relative error at most 2^-23) instead of the correctly
// rounded root, whose multi-instruction sequence took a third of the loop.
__device__ __forceinline__ F2 nrmse_term2(F2 G, F2 sg, F2 sg2, F2 qs, const EpiConsts& ec) {
  const F2 one = f2(1.0f, 1.0f), sc = f2(ec.nrmse_scale, ec.nrmse_scale);
  const F2 ds = sub2(sg, qs);
  float x0, x1;
  f2_split(mul2(sc, fma2(ds, ds, mul2(mul2(sg2, qs), sub2(one, G)))), x0, x1);
  return f2(sqrt_approx(fmaxf(x0, 0.0f)), sqrt_approx(fmaxf(x1, 0.0f)));
}

// Pairwise form: numerator factor x and weight w of two pairs; the term is x w
// for the weighted metrics and x for unweighted NRMSE (2D) and the diagnostic
// metrics. Same arithmetic as pair_terms.
template <int METRIC, bool EXACT>
__device__ __forceinline__ void terms2(F2 G, const RowC& rc, F2 qa, F2 qr, F2 qs, F2 qm, const EpiConsts& ec,
                                       F2& x, F2& w) {
  const F2 one = f2(1.0f, 1.0f);
  if (METRIC == kDebugDot) {
    x = mul2(G, mul2(rc.a, qa));
    return;
  }
  if (METRIC == kDebugSum) {
    x = add2(rc.r, qr);
    return;
  }
  if (METRIC == kNrmse) {
    x = nrmse_term2(G, rc.sg, rc.sg2, qs, ec);
    return;
  }
  const F2 d = sub2(rc.a, qa);
  float m0, m1;
  f2_split(mul2(d, d), m0, m1);
  w = f2(ex2_approx(-m0), ex2_approx(-m1));
  float x0, x1;
  if (METRIC == kPearson) {
    F2 gc;
    if (!EXACT) {
      gc = fma2(mul2(G, rc.ne), qr, G);  // G (1 - t)
    } else {
      float d0, d1;
      f2_split(sub2(one, mul2(rc.ne, qr)), d0, d1);  // 1 + t
      gc = mul2(G, f2(rcp_approx(d0), rcp_approx(d1)));
    }
    f2_split(gc, x0, x1);
    x = f2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f));
  } else if (METRIC == kSsim) {
    const F2 c1 = f2(ec.c1, ec.c1), c2 = f2(ec.c2, ec.c2);
    const F2 num = mul2(fma2(rc.mu2, qm, c1), fma2(mul2(rc.sg2, qs), G, c2));
    const F2 den = mul2(fma2(rc.mumu, mul2(qm, qm), c1), fma2(qs, qs, rc.s2));
    float e0, e1, q0, q1;
    f2_split(den, e0, e1);
    f2_split(mul2(num, f2(rcp_approx(e0), rcp_approx(e1))), q0, q1);
    x = f2(fmaxf(q0, 0.0f), fmaxf(q1, 0.0f));
  } else {  // kNrmseW
    x = nrmse_term2(G, rc.sg, rc.sg2, qs, ec);
  }
}

// Exact squared distance of two FP32 unit vectors (NRMSE near-identical pairs).
__device__ __noinline__ float exact_diff2(const float* __restrict__ up, const float* __restrict__ uq, int K) {
  float acc = 0.0f;
  for (int i = 0; i < K; i++) {
    const float d = up[i] - uq[i];
    acc = fmaf(d, d, acc);
  }
  return acc;
}

// Correction of a near-identical NRMSE pair: the term of the exact squared
// difference minus the one nrmse_term2 added (recomputed with its arithmetic).
__device__ __noinline__ float nrmse_correction(float g, float sp, float sq, int p, int q, const float* __restrict__ U,
                                               int kp, int K, float scale) {
  const float ds = __fsub_rn(sp, sq);
  const float approx = sqrt_approx(fmaxf(
      __fmul_rn(scale, __fmaf_rn(ds, ds, __fmul_rn(__fmul_rn(__fadd_rn(sp, sp), sq), __fsub_rn(1.0f, g)))), 0.0f));
  const float D = (q == p) ? 0.0f : exact_diff2(U + (size_t)p * kp, U + (size_t)q * kp, K);
  return sqrtf(__fmul_rn(scale, __fmaf_rn(ds, ds, __fmul_rn(__fmul_rn(sp, sq), D)))) - approx;
}

__device__ __forceinline__ void f2_add_half(F2& v, int half, float x) {
  float lo, hi;
  f2_split(v, lo, hi);
  if (half) hi += x;
  else lo += x;
  v = f2(lo, hi);
}

// A warp's part of a tile, a slab: 32 rows x W columns, in chunks of 16
// columns, each read for both 16-lane halves of the warp's 32 TMEM lanes. Each thread has 4
// rows (32(w%4) + t/4 + 8k) and 4 columns per chunk (2(t%4) + {0, 1}, 8 + 2(t%4) +
// {0, 1}). rs: the tile's row parameters; cs: the slab's column parameters
// (permuted); cacc[c][rep]: the item's column sums of this thread, in registers;
// p0: block index of tile row 0; q0: of the slab's first column; fs: this warp's
// scratch (f by row, then g by permuted column). Row sums go to rsum[k].
//
// Row and column factors of the slab: row 32(w%4) + lane and columns (permuted
// positions) lane + 32 j of this lane. They need no accumulator, so they are
// computed while its MMAs run.
template <int METRIC>
__device__ __forceinline__ void slab_factors(const float* __restrict__ rs, const float* __restrict__ cs,
                                             const SlabC& sc, float* __restrict__ fs, const EpiConsts& ec) {
  const int lane = threadIdx.x & 31;
  const int row = (threadIdx.x & 96) + lane;
  const float sa = sc.alpha * ec.inv_wscale, sb = sc.beta * ec.inv_wscale;
  const float a = rs[row], d = a - sc.beta;
  float f = ex2_approx(fmaf(-d, d, sc.sf * (a - sc.alpha))) * sc.cf;
  if (METRIC == kSsim) {
    const float s = rs[kRowS + row];
    f *= 2.0f * s * rcp_approx(fmaf(s, s, fmaf(sb, sb, ec.c2)));
  }
  fs[(lane & 7) * 4 + (lane >> 3)] = f;
  const float S = fmaf(sa, sa, fmaf(sb, sb, ec.c2));
#pragma unroll
  for (int j = 0; j < Cfg<METRIC>::kColW / 32; j++) {
    const int i = lane + 32 * j;
    const float dq = cs[i] - sc.beta;
    float g = ex2_approx(dq * (sc.eg - dq));
    if (METRIC == kSsim) {
      const float s = cs[2 * kBN + i];
      g *= s * S * rcp_approx(fmaf(s, s, fmaf(sa, sa, ec.c2)));
    }
    fs[32 + i] = g;
  }
}

// The slab's pair loop (FIRST: with the first-order weight factor per pair;
// unweighted NRMSE has no factors). TMEM is read 16 columns at a time, the next
// 16 issued before the current ones are evaluated.
template <int METRIC, bool FIRST>
__device__ __forceinline__ void tile_factor(uint32_t taddr, const float* __restrict__ rs, const float* __restrict__ cs,
                                            const SlabC& sc, const float* __restrict__ fs,
                                            F2 (&cacc)[Cfg<METRIC>::kCH][2], const EpiConsts& ec, int p0, int q0,
                                            float (&rsum)[4]) {
  constexpr int CH = Cfg<METRIC>::kCH;
  constexpr bool WGT = weighted_num<METRIC>();
  const int lane = threadIdx.x & 31, rsub = lane >> 2, csub = lane & 3;
  const int quarter = (threadIdx.x >> 5) & 3;
  uint32_t buf[2][2][8];
  tmem_ld_batch(taddr, buf[0]);
  F2 fr[4], rn[4], dp[4], mu[4], rr[4], sg[4];
  if (WGT) {
    const float4 f4 = *reinterpret_cast<const float4*>(fs + 4 * rsub);
    fr[0] = f2(f4.x, f4.x);
    fr[1] = f2(f4.y, f4.y);
    fr[2] = f2(f4.z, f4.z);
    fr[3] = f2(f4.w, f4.w);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    rn[k] = f2(0.0f, 0.0f);
    const int row = quarter * 32 + rsub + 8 * k;
    if (FIRST) {
      const float v = sc.kc * (rs[row] - sc.alpha);
      dp[k] = f2(v, v);
    }
    if (METRIC == kSsim) {
      const float m = rs[kRowMu + row], r = ec.c2h * rs[kRowR + row];
      mu[k] = f2(m, m);
      rr[k] = f2(r, r);
    }
    if (nrmse_tc<METRIC>()) {
      const float v = rs[kRowS + row];
      sg[k] = f2(v, v);
    }
  }
  tmem_wait_batch(buf[0]);
#pragma unroll
  for (int c = 0; c < CH; c++) {
    uint32_t(&cur)[2][8] = buf[c & 1];
    uint32_t(&nxt)[2][8] = buf[(c + 1) & 1];
    if (c + 1 < CH) tmem_ld_batch(taddr + 16 * (c + 1), nxt);
    {
      const int cb = 16 * c + 4 * csub;
      float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f), r4 = g4, s4 = g4, m4 = g4, a4 = g4;
      if (WGT) g4 = *reinterpret_cast<const float4*>(fs + 32 + cb);
      if (FIRST) a4 = *reinterpret_cast<const float4*>(cs + cb);
      if (METRIC == kSsim) {
        r4 = *reinterpret_cast<const float4*>(cs + kBN + cb);
        m4 = *reinterpret_cast<const float4*>(cs + 3 * kBN + cb);
      }
      if (nrmse_tc<METRIC>()) s4 = *reinterpret_cast<const float4*>(cs + 2 * kBN + cb);
      const F2 qg[2] = {f2(g4.x, g4.y), f2(g4.z, g4.w)};
      F2 cn[2] = {f2(0.0f, 0.0f), f2(0.0f, 0.0f)};
      float near = 1.0f;  // NRMSE: smallest 1 - G
#pragma unroll
      for (int rep = 0; rep < 2; rep++) {
        const F2 dq = FIRST ? sub2(rep ? f2(a4.z, a4.w) : f2(a4.x, a4.y), f2(sc.beta, sc.beta))
                            : f2(0.0f, 0.0f);
        const F2 qr = rep ? f2(r4.z, r4.w) : f2(r4.x, r4.y);
        const F2 qs = rep ? f2(s4.z, s4.w) : f2(s4.x, s4.y);
        const F2 qm = rep ? f2(m4.z, m4.w) : f2(m4.x, m4.y);
#pragma unroll
        for (int kr = 0; kr < 4; kr++) {
          const int vi = 4 * rep + 2 * (kr & 1);
          const float g0 = __uint_as_float(cur[kr >> 1][vi]), g1 = __uint_as_float(cur[kr >> 1][vi + 1]);
          F2 x;
          if (METRIC == kPearson) {
            x = f2(fmaxf(g0, 0.0f), fmaxf(g1, 0.0f));
          } else if (METRIC == kSsim) {
            const F2 c1 = f2(ec.c1, ec.c1), two = f2(2.0f, 2.0f);
            const F2 m = mul2(mu[kr], qm);
            float e0, e1, x0, x1;
            f2_split(fma2(m, m, c1), e0, e1);
            const F2 y = mul2(fma2(rr[kr], qr, f2(g0, g1)), fma2(m, two, c1));
            f2_split(mul2(y, f2(rcp_approx(e0), rcp_approx(e1))), x0, x1);
            x = f2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f));
          } else {
            const F2 G = mul2(f2(g0, g1), f2(ec.gscale, ec.gscale));
            float t0, t1;
            f2_split(G, t0, t1);
            near = min3(near, 1.0f - t0, 1.0f - t1);
            x = nrmse_term2(G, sg[kr], add2(sg[kr], sg[kr]), qs, ec);
          }
          if (FIRST) x = fma2(mul2(x, dp[kr]), dq, x);
          if (WGT) {
            rn[kr] = fma2(x, qg[rep], rn[kr]);
            cn[rep] = kr == 0 ? mul2(x, fr[kr]) : fma2(x, fr[kr], cn[rep]);
          } else {
            rn[kr] = add2(rn[kr], x);
            cn[rep] = kr == 0 ? x : add2(cn[rep], x);
          }
        }
      }
      if (nrmse_tc<METRIC>() && near < 1.0f - ec.nrmse_near) {
        // Near-identical pairs: replace the accumulated term by the one of the
        // exact squared difference.
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int rep = j >> 3, kr = (j >> 1) & 3, lh = j & 1;
          const float g = __fmul_rn(__uint_as_float(cur[kr >> 1][4 * rep + 2 * (kr & 1) + lh]), ec.gscale);
          if (!(g > ec.nrmse_near)) continue;
          const int row = quarter * 32 + rsub + 8 * kr, q = q0 + 16 * c + 8 * rep + 2 * csub + lh;
          const int ci = 16 * c + 4 * csub + 2 * rep + lh;  // permuted column slot
          float corr = nrmse_correction(g, rs[kRowS + row], cs[2 * kBN + ci], p0 + row, q, ec.U, ec.kp, ec.K,
                                        ec.nrmse_scale);
          if (FIRST) corr = fmaf(corr * sc.kc * (rs[row] - sc.alpha), cs[ci] - sc.beta, corr);
          float glo = 1.0f, ghi = 1.0f, flo = 1.0f, fhi;
          if (WGT) {
            f2_split(qg[rep], glo, ghi);
            f2_split(fr[kr], flo, fhi);
          }
          f2_add_half(rn[kr], lh, corr * (lh ? ghi : glo));
          f2_add_half(cn[rep], lh, corr * flo);
        }
      }
#pragma unroll
      for (int rep = 0; rep < 2; rep++)
        cacc[c][rep] = WGT ? fma2(cn[rep], qg[rep], cacc[c][rep]) : add2(cn[rep], cacc[c][rep]);
    }
    if (c + 1 < CH) tmem_wait_batch(nxt);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    float lo, hi;  // f is applied to the reduced row sums
    f2_split(rn[k], lo, hi);
    rsum[k] = lo + hi;
  }
}

// Pairwise form. Row passes: the metrics with many row constants (SSIM, NRMSE)
// take the 4 rows in two passes of 2 so that their constants fit in registers.
template <int METRIC>
constexpr int row_passes() {
  return (METRIC == kSsim || METRIC == kNrmse || METRIC == kNrmseW) ? 2 : 1;
}

template <int METRIC, bool EXACT, bool MASKED>
__device__ __forceinline__ void tile_pairs(uint32_t taddr, const float* __restrict__ rs, const float* __restrict__ cs,
                                           F2 (&cacc)[Cfg<METRIC>::kCH][2], int p0, int q0, const EpiConsts& ec,
                                           float (&rsum)[4]) {
  constexpr int CH = Cfg<METRIC>::kCH;
  constexpr int NP = row_passes<METRIC>(), R = 4 / NP;  // passes, rows per pass
  constexpr int HP = R / 2;                              // 16-lane halves per pass
  const int lane = threadIdx.x & 31, rsub = lane >> 2, csub = lane & 3;
  const int quarter = (threadIdx.x >> 5) & 3;
#pragma unroll 1
  for (int pass = 0; pass < NP; pass++) {
    RowC rc[R];
    F2 rn[R];
    int prow[R];
    bool force[R];
#pragma unroll
    for (int kr = 0; kr < R; kr++) {
      const int row = quarter * 32 + rsub + 8 * (pass * R + kr);
      rc[kr] = make_rowc<METRIC>(rs, row, ec);
      rn[kr] = f2(0.0f, 0.0f);
      prow[kr] = p0 + row;
      force[kr] = MASKED && rs[kRowR + row] > 0.0f;
    }
    // TMEM reads, one (chunk, half) step at a time; the next step's load is
    // issued before the current step is evaluated.
    const uint32_t tp = taddr + ((uint32_t)(16 * pass * HP) << 16);
    uint32_t buf[2][8];
    tmem_ld8(tp, buf[0]);
    tmem_wait8(buf[0]);
#pragma unroll
    for (int c = 0; c < CH; c++) {
      const int cb = 16 * c + 4 * csub;
      float4 a4 = make_float4(0.f, 0.f, 0.f, 0.f), r4 = a4, s4 = a4, m4 = a4;
      if (METRIC != kNrmse && METRIC != kDebugSum) a4 = *reinterpret_cast<const float4*>(cs + cb);
      if (METRIC == kPearson || METRIC == kDebugSum) r4 = *reinterpret_cast<const float4*>(cs + kBN + cb);
      if (METRIC == kSsim || nrmse_tc<METRIC>()) s4 = *reinterpret_cast<const float4*>(cs + 2 * kBN + cb);
      if (METRIC == kSsim) m4 = *reinterpret_cast<const float4*>(cs + 3 * kBN + cb);
#pragma unroll
      for (int hh = 0; hh < HP; hh++) {
        const int step = c * HP + hh;
        uint32_t(&cur)[8] = buf[step & 1];
        uint32_t(&nxt)[8] = buf[(step + 1) & 1];
        if (step + 1 < CH * HP) {
          const int nc = (step + 1) / HP, nh = (step + 1) % HP;
          tmem_ld8(tp + ((uint32_t)(16 * nh) << 16) + 16 * nc, nxt);
        }
        float near = 1.0f;  // NRMSE: smallest 1 - G
#pragma unroll
        for (int rep = 0; rep < 2; rep++) {
          const F2 qa = rep ? f2(a4.z, a4.w) : f2(a4.x, a4.y);
          const F2 qr = rep ? f2(r4.z, r4.w) : f2(r4.x, r4.y);
          const F2 qs = rep ? f2(s4.z, s4.w) : f2(s4.x, s4.y);
          const F2 qm = rep ? f2(m4.z, m4.w) : f2(m4.x, m4.y);
          const int qlo = q0 + 16 * c + 8 * rep + 2 * csub;
#pragma unroll
          for (int kk = 0; kk < 2; kk++) {
            const int kr = 2 * hh + kk;
            F2 G = mul2(f2(__uint_as_float(cur[4 * rep + 2 * kk]), __uint_as_float(cur[4 * rep + 2 * kk + 1])),
                        f2(ec.gscale, ec.gscale));
            const int p = prow[kr];
            if (MASKED) {
              float g0, g1;
              f2_split(G, g0, g1);
              if (force[kr] && qlo == p) g0 = 1.0f;
              if (force[kr] && qlo + 1 == p) g1 = 1.0f;
              G = f2(g0, g1);
            }
            F2 x, w;
            terms2<METRIC, EXACT>(G, rc[kr], qa, qr, qs, qm, ec, x, w);
            if (nrmse_tc<METRIC>()) {
              float g0, g1;
              f2_split(G, g0, g1);
              near = min3(near, 1.0f - g0, 1.0f - g1);
            }
            if (!MASKED) {
              if (weighted_num<METRIC>()) {
                rn[kr] = fma2(x, w, rn[kr]);
                cacc[c][rep] = fma2(x, w, cacc[c][rep]);
              } else {
                rn[kr] = add2(rn[kr], x);
                cacc[c][rep] = add2(cacc[c][rep], x);
              }
            } else {
              float x0, x1;
              f2_split(weighted_num<METRIC>() ? mul2(x, w) : x, x0, x1);
              const bool pv = p < ec.n;
              const bool r0 = pv && qlo >= p && qlo < ec.n, r1 = pv && qlo + 1 >= p && qlo + 1 < ec.n;
              const bool c0 = r0 && qlo != p, c1 = r1 && qlo + 1 != p;
              rn[kr] = add2(rn[kr], f2(r0 ? x0 : 0.0f, r1 ? x1 : 0.0f));
              cacc[c][rep] = add2(cacc[c][rep], f2(c0 ? x0 : 0.0f, c1 ? x1 : 0.0f));
            }
          }
        }
        if (nrmse_tc<METRIC>() && near < 1.0f - ec.nrmse_near) {
          // Near-identical pairs: replace the accumulated term by the one of the
          // exact squared difference.
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int rep = j >> 2, kk = (j >> 1) & 1, lh = j & 1;
            const int kr = 2 * hh + kk;
            const float g = __fmul_rn(__uint_as_float(cur[4 * rep + 2 * kk + lh]), ec.gscale);
            const int row = quarter * 32 + rsub + 8 * (pass * R + kr);
            const int p = prow[kr], q = q0 + 16 * c + 8 * rep + 2 * csub + lh;
            const bool rv = !MASKED || (p < ec.n && q >= p && q < ec.n);
            const bool cv = !MASKED || (rv && q != p);
            float ge = g;
            if (MASKED && force[kr] && q == p) ge = 1.0f;
            if (!(ge > ec.nrmse_near) || !rv) continue;
            const int ci = 16 * c + 4 * csub + 2 * rep + lh;  // permuted column slot
            float corr = nrmse_correction(ge, rs[kRowS + row], cs[2 * kBN + ci], p, q, ec.U, ec.kp, ec.K, ec.nrmse_scale);
            if (METRIC == kNrmseW) {
              const float d = __fsub_rn(rs[row], cs[ci]);
              corr *= ex2_approx(-__fmul_rn(d, d));
            }
            f2_add_half(rn[kr], lh, corr);
            if (cv) f2_add_half(cacc[c][rep], lh, corr);
          }
        }
        if (step + 1 < CH * HP) tmem_wait8(nxt);
      }
    }
#pragma unroll
    for (int kr = 0; kr < R; kr++) {
      float lo, hi;
      f2_split(rn[kr], lo, hi);
      // compile-time indices into rsum (the pass loop is not unrolled)
      if (pass == 0) rsum[kr] = lo + hi;
      else rsum[(NP - 1) * R + kr] = lo + hi;
    }
  }
}

// Row sums of the 4 lanes that share rows (lanes 4i..4i+3): x[k] holds row k's
// partial; lane t ends with row k = 2 (t & 1) + ((t >> 1) & 1).
__device__ __forceinline__ float reduce_rows4(const float (&x)[4]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2;
  float y[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float keep = b0 ? x[2 + i] : x[i], send = b0 ? x[i] : x[2 + i];
    y[i] = keep + __shfl_xor_sync(full, send, 1);
  }
  const float keep = b1 ? y[1] : y[0], send = b1 ? y[0] : y[1];
  return keep + __shfl_xor_sync(full, send, 2);
}

// Column sums of the 8 lanes that share columns (lanes with equal t % 4),
// then one FP64 atomic add per column. x index: (c * 2 + rep) * 2 + lohi,
// column 16c + 8rep + 2(t % 4) + lohi.
template <int NV>
__device__ __forceinline__ void flush_columns(const float (&x)[NV], int q0, const EpiConsts& ec, double* num) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, csub = lane & 3;
  const int b1 = (lane >> 2) & 1, b2 = (lane >> 3) & 1, b3 = (lane >> 4) & 1;
  float y[NV / 2], z[NV / 4], u[NV / 8];
#pragma unroll
  for (int i = 0; i < NV / 2; i++) {
    const float keep = b1 ? x[NV / 2 + i] : x[i], send = b1 ? x[i] : x[NV / 2 + i];
    y[i] = keep + __shfl_xor_sync(full, send, 4);
  }
#pragma unroll
  for (int i = 0; i < NV / 4; i++) {
    const float keep = b2 ? y[NV / 4 + i] : y[i], send = b2 ? y[i] : y[NV / 4 + i];
    z[i] = keep + __shfl_xor_sync(full, send, 8);
  }
#pragma unroll
  for (int i = 0; i < NV / 8; i++) {
    const float keep = b3 ? z[NV / 8 + i] : z[i], send = b3 ? z[i] : z[NV / 8 + i];
    u[i] = keep + __shfl_xor_sync(full, send, 16);
  }
#pragma unroll
  for (int j = 0; j < NV / 8; j++) {
    const int i = b1 * (NV / 2) + b2 * (NV / 4) + b3 * (NV / 8) + j;
    const int c = i >> 2, rep = (i >> 1) & 1, lohi = i & 1;
    const int q = q0 + 16 * c + 8 * rep + 2 * csub + lohi;
    if (q < ec.n) atomicAdd(num + q, (double)u[j]);
  }
}

// Work items. Run j holds row blocks [jL, jL + L); it meets the column tiles
// ct >= j h (h = L / (BN / 128): the first column tile that reaches the run's
// rows), each (run, column tile) an item, clipped to the triangle. The column
// tiles are grouped into panels of g.panel tiles whose B operand fits in L2;
// items go panel by panel, within a panel run by run, within a run by column
// tile. All CTAs then work on the same row blocks at once (their A tiles are
// read from DRAM once per panel and shared in L2), and a panel's B tiles stay
// in L2 while every run passes over them (B is read from DRAM about once).
// With one panel this is the plain run-major order.
//
// Items of runs [0, j) in the panel of column tiles [c0, c1): sum over
// j' < j of c1 - max(c0, j' h).
__host__ __device__ inline long long panel_items_before_run(long long j, int c0, int c1, int h) {
  const long long a = min(j, (long long)(c0 / h) + 1);  // runs with j' h <= c0 take the whole panel
  long long s = a * (c1 - c0);
  if (j > a) s += (j - a) * (long long)c1 - (long long)h * (j * (j - 1) / 2 - a * (a - 1) / 2);
  return s;
}

// Items of runs [0, j) over all column tiles (one panel).
__host__ __device__ inline long long items_before_run(long long j, int n_ct, int h) {
  return j * n_ct - (long long)h * j * (j - 1) / 2;
}

// Runs that reach the panel [c0, c1) (j h <= c1 - 1), at most n_runs.
__host__ __device__ inline int panel_runs(int c1, int h, int n_runs) { return min((c1 - 1) / h + 1, n_runs); }

// Item -> (column tile, row-block range); false for an empty range.
__host__ __device__ inline bool decode_item(long long it, const TcArgs& g, int m, int& ct, int& rb0, int& rb1) {
  long long base = 0;
  int c0 = 0, c1 = 0, J = 0;
  for (int k = 0; k < g.n_panels; k++) {
    c0 = k * g.panel;
    c1 = min(c0 + g.panel, g.n_ct);
    J = panel_runs(c1, g.h, g.n_runs);
    const long long cnt = panel_items_before_run(J, c0, c1, g.h);
    if (it < base + cnt || k == g.n_panels - 1) break;
    base += cnt;
  }
  const long long r = it - base;
  int lo = 0, hi = J - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (panel_items_before_run(mid, c0, c1, g.h) <= r) lo = mid;
    else hi = mid - 1;
  }
  ct = max(c0, lo * g.h) + (int)(r - panel_items_before_run(lo, c0, c1, g.h));
  rb0 = lo * g.L;
  rb1 = min(rb0 + g.L, min((ct + 1) * m, g.n_rb));
  return rb0 < rb1 && ct < c1;
}

// A CTA's walk over its items it = start, start + stride, ...: the first is
// decoded with decode_item's search, each later one by stepping forward run by
// run (a few operations per step instead of a search per item, which matters
// for small maps whose items hold few tiles).
struct ItemCursor {
  long long it;  // current item
  long long r;   // its offset among the items of run j in panel k
  int k, c0, c1, J, j;

  __host__ __device__ __forceinline__ void set_panel(const TcArgs& g, int kk) {
    k = kk;
    c0 = kk * g.panel;
    c1 = min(c0 + g.panel, g.n_ct);
    J = panel_runs(c1, g.h, g.n_runs);
  }
  __host__ __device__ __forceinline__ void init(const TcArgs& g, long long start) {
    it = start;
    long long base = 0;
    set_panel(g, 0);
    while (k < g.n_panels - 1) {
      const long long cnt = panel_items_before_run(J, c0, c1, g.h);
      if (start < base + cnt) break;
      base += cnt;
      set_panel(g, k + 1);
    }
    const long long rr = start - base;
    int lo = 0, hi = J - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (panel_items_before_run(mid, c0, c1, g.h) <= rr) lo = mid;
      else hi = mid - 1;
    }
    j = lo;
    r = rr - panel_items_before_run(lo, c0, c1, g.h);
  }
  __host__ __device__ __forceinline__ void advance(const TcArgs& g, long long d) {
    it += d;
    r += d;
    for (;;) {
      const int cnt = c1 - max(c0, j * g.h);  // >= 1 for every run below J
      if (r < cnt) break;
      r -= cnt;
      if (++j >= J) {
        if (k + 1 >= g.n_panels) break;  // past the last item; the caller stops on it
        set_panel(g, k + 1);
        j = 0;
      }
    }
  }
  // The tiles of the current item that pass `phase` takes: pass 0 the full
  // tiles, pass 1 the masked ones (tiles that reach the diagonal, rb >= ct m,
  // and every tile of a ragged last column tile). Every role walks pass 0 over
  // all of the CTA's items, then pass 1, so the masked epilogue runs in a loop
  // of its own. False for an empty range.
  __host__ __device__ __forceinline__ bool part(const TcArgs& g, int m, int bn, int phase, int& ct, int& lo,
                                                int& hi) const {
    ct = max(c0, j * g.h) + (int)r;
    const int rb0 = j * g.L, rb1 = min(rb0 + g.L, min((ct + 1) * m, g.n_rb));
    const bool full = (long long)(ct + 1) * bn <= g.ec.n;
    const int rbm = full ? min(max(rb0, ct * m), rb1) : rb0;
    lo = phase == 0 ? rb0 : rbm;
    hi = phase == 0 ? rbm : rb1;
    return lo < hi;
  }
};

template <int CTAS>
__device__ __forceinline__ ItemCursor first_item(const TcArgs& g) {
  ItemCursor c;
  c.init(g, g.item0 + blockIdx.x / CTAS);
  return c;
}

template <int CTAS>
__device__ __forceinline__ void group_sync() {
  if constexpr (CTAS == 2) cluster_sync();
  else __syncthreads();
}

// Ring stage of a tile's last operands: st0 is the stage of its first ones, back =
// (stages per tile - 1) % S. (A tile may take more stages than the ring has: K = 197 takes
// seven of a ring of five.)
__host__ __device__ inline uint32_t ring_last(uint32_t st0, uint32_t back, uint32_t S) {
  const uint32_t s = st0 + back;  // both below S
  return s < S ? s : s - S;
}

// End of a role: all warps (of both CTAs of a pair) meet (no CTA leaves while the
// other may still arrive on its barriers or an MMA reads its shared memory), then
// the MMA warps free TMEM.
template <int CTAS>
__device__ __forceinline__ void role_exit(uint32_t tmem, bool owner) {
  tc_fence_before();
  group_sync<CTAS>();
  tc_fence_after();
  if (!owner) return;
  if constexpr (CTAS == 2)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kBN) : "memory");
  else
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kBN) : "memory");
}

template <int METRIC, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kThreads, 1)
    k_gram_tc(const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmB, TcArgs g) {
  using C = Cfg<METRIC>;
  constexpr int CH = C::kCH, EW = kEpiWarps, W = C::kColW, SETS = C::kSets;
  constexpr int M = CTAS;            // row blocks per tile
  constexpr int BH = 2 / CTAS;       // halves of the column tile in this CTA
  extern __shared__ __align__(1024) uint8_t sbase[];  // (swizzled tiles need 1,024-byte alignment)
  const uint32_t base = smem_u32(sbase);
  const int S = g.stages;
  const uint32_t rank = CTAS == 2 ? blockIdx.x & 1 : 0, n_clusters = gridDim.x / CTAS;
  const uint32_t stage_bytes = (uint32_t)g.sc * kChunkBytes;
  const uint32_t sB = base;                                            // this CTA's part of the column tile
  const uint32_t sA = sB + BH * g.nch * kChunkBytes;                   // S stages of row-block chunks
  const uint32_t sC = sA + S * stage_bytes;                            // 2 column-parameter slots
  const uint32_t sR = sC + 2 * kColFloats * 4;                         // kRSlots row-parameter slots
  const uint32_t sF = sR + kRSlots * kRowFloats * 4;                   // f and g of each epilogue warp
  const uint32_t sBar = sF + EW * kScratch * 4;
  const float* cslots = reinterpret_cast<const float*>(sbase + (sC - base));
  const float* rslots = reinterpret_cast<const float*>(sbase + (sR - base));
  float* scratch = reinterpret_cast<float*>(sbase + (sF - base));
  // barriers: a_full[16], a_empty[16], b_full, b_empty, acc_full[2], acc_empty[2],
  //           c_full[2], c_empty[2], r_full[4], r_empty[4], done; then the TMEM
  //           address
  const uint32_t b_afull = sBar, b_aempty = b_afull + 8 * kMaxStages, b_bfull = b_aempty + 8 * kMaxStages,
                 b_bempty = b_bfull + 8, b_accf = b_bempty + 8, b_acce = b_accf + 16, b_cfull = b_acce + 16,
                 b_cempty = b_cfull + 16, b_rfull = b_cempty + 16, b_rempty = b_rfull + 8 * kRSlots,
                 b_done = b_rempty + 8 * kRSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sbase + (b_done + 8 - base));

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (warp: uniform)
  if (threadIdx.x == 0) {
    // operand barriers of CTA 0: its own producer and CTA 1's relay
    const uint32_t full = CTAS == 2 && rank == 0 ? 2 : 1;
    for (int s = 0; s < kMaxStages; s++) {
      mbar_init(b_afull + 8 * s, full);
      mbar_init(b_aempty + 8 * s, 1);
    }
    mbar_init(b_bfull, full);
    mbar_init(b_bempty, 1);
    for (int b = 0; b < 2; b++) {
      mbar_init(b_accf + 8 * b, 1);
      mbar_init(b_acce + 8 * b, CTAS * EW / SETS);  // (CTA 0's: the epilogue warps of both CTAs)
      mbar_init(b_cfull + 8 * b, 1);
      mbar_init(b_cempty + 8 * b, EW);
    }
    for (int r = 0; r < kRSlots; r++) {
      mbar_init(b_rfull + 8 * r, 1);
      mbar_init(b_rempty + 8 * r, EW / SETS);
    }
    mbar_init(b_done, 1);
    if (base & 1023) atomicCAS(g.status, ST_OK, ST_ALIGNMENT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Operand offsets (16-byte units, within a stage and the column tile) of the
  // tile's MMAs. A block of 16 fp16 is 32 B, four to a chunk. Row part P meets the column parts
  // 0 .. parts - 1 - P, in the order of the row operand's blocks: hi with hi and mid, mid with
  // hi, row tails with column tails. Every MMA truncates the accumulator, so the products of
  // three parts go smallest first where one stage holds the tile (5x5 Pearson: numerators off
  // by -1.6e-7 +- 4.8e-8 in the order of the blocks, by -4.7e-8 +- 4.0e-8 so; two parts: 9x9
  // SSIM takes 1% longer so).
  uint2* mma_tab = reinterpret_cast<uint2*>(sbase + (sBar + kBarBytes - base));
  uint32_t* mma_end = reinterpret_cast<uint32_t*>(mma_tab + kMaxMma);  // MMAs up to the end of each stage
  if (warp == 2) {
    const int parts = g.parts, nb = g.nb, nt = g.nt, n_full = parts * (parts + 1) / 2 * nb, n = n_full + nt;
    constexpr uint32_t kChunkU = kChunkBytes >> 4;
    for (int m = lane; m <= n; m += 32) {  // (entry n: read ahead, never used)
      int qa = 0, qb = 0;
      if (parts == 3 && g.nst == 1) {
        if (m >= n - nb && m < n) {  // hi.hi
          qa = qb = m - (n - nb);
        } else if (m >= n_full - nb) {
          qa = parts * nb + min(m - (n_full - nb), max(nt - 1, 0));
          qb = qa + nt;
        } else {
          int s = parts - 1, i = m;  // the products of parts P + Q = s
          while (i >= (s + 1) * nb) i -= (s + 1) * nb, s--;
          qa = i / nb * nb + i % nb;
          qb = (s - i / nb) * nb + i % nb;
        }
      } else if (m < n_full) {
        int P = 0, i = m;
        while (i >= (parts - P) * nb) i -= (parts - P) * nb, P++;
        qa = P * nb + i / (parts - P);
        qb = i % (parts - P) * nb + i / (parts - P);
      } else {
        qa = parts * nb + min(m - n_full, max(nt - 1, 0));
        qb = qa + nt;
      }
      const uint32_t ca = (uint32_t)(qa >> 2) % (uint32_t)g.sc, cb = (uint32_t)(qb >> 2);
      mma_tab[m] = make_uint2(ca * kChunkU + 2 * (qa & 3), cb * (BH * kChunkU) + 2 * (qb & 3));
    }
    for (int st = lane; st < g.nst; st += 32) {
      int q = min(parts * nb + nt, 4 * (st + 1) * g.sc), m = max(q - parts * nb, 0);
      for (int P = 0; P < parts; P++) m += (parts - P) * min(max(q - P * nb, 0), nb);
      mma_end[st] = m;
    }
  }
  if (warp == 1) {  // the MMA warps of both CTAs own the TMEM allocation
    if constexpr (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"(2 * kBN)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"(2 * kBN)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  group_sync<CTAS>();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA
    if (lane == 0) {
      long long tile = 0;
      uint32_t item_i = 0, n_r = 0, n_a = 0;  // items, row-parameter loads, stage loads issued
      uint32_t s = 0, eph = 0;                // ring: stage, parity of the round being refilled
      bool ok = true;
      for (int phase = 0; ok && phase < 2; phase++)
      for (ItemCursor cur = first_item<CTAS>(g); ok && cur.it < g.item1; cur.advance(g, n_clusters)) {
        int ct, rb0, rb1;
        if (!cur.part(g, kBN / kBM, kBN, phase, ct, rb0, rb1)) continue;
        const uint32_t cs = item_i & 1;
        // the column-parameter slot the epilogue released two items ago, and the
        // B buffer once the MMAs of the previous item are complete
        if (!mbar_wait(b_cempty + 8 * cs, ((item_i >> 1) & 1) ^ 1, g, ST_TIMEOUT_PRODUCER, true, true)) { ok = false; break; }
        if (item_i > 0 && !mbar_wait(b_bempty, (item_i - 1) & 1, g, ST_TIMEOUT_PRODUCER, true, true)) { ok = false; break; }
        mbar_expect_tx(b_bfull, BH * g.nch * kChunkBytes);
        const int yb = ct * kBN + (int)rank * kBM;
        for (int c = 0; c < g.nch; c += g.sc) tma_load_3d(sB + BH * c * kChunkBytes, &tmB, b_bfull, yb, c);
        mbar_expect_tx(b_cfull + 8 * cs, kColFloats * 4);
        bulk_load(sC + cs * kColFloats * 4, g.colsoa + (size_t)ct * kColFloats, kColFloats * 4, b_cfull + 8 * cs);
        item_i++;
        {  // the B tile of this cluster's next item into L2
          int nct, nrb0, nrb1;
          ItemCursor nx = cur;
          nx.advance(g, n_clusters);
          if (nx.it < g.item1 && nx.part(g, kBN / kBM, kBN, phase, nct, nrb0, nrb1) && nct != ct)
            for (int c = 0; c < g.nch; c += g.sc) tma_prefetch_3d(&tmB, nct * kBN + (int)rank * kBM, c);
        }
        for (int rb = rb0; ok && rb < rb1; rb += M, tile++) {
          if (tile == g.withhold) { ok = false; break; }
          const int ya = (rb + (int)rank) * kBM;
          for (int st = 0; st < g.nst; st++) {
            // stage s is free once the MMAs that read it are complete
            if (!mbar_wait(b_aempty + 8 * s, eph ^ 1, g, ST_TIMEOUT_PRODUCER, true, true)) { ok = false; break; }
            mbar_expect_tx(b_afull + 8 * s, stage_bytes);
            tma_load_3d(sA + s * stage_bytes, &tmU, b_afull + 8 * s, ya, st * g.sc);
            n_a++;
            if (++s == (uint32_t)S) {
              s = 0;
              eph ^= 1;
            }
          }
          if (!ok) break;
          const uint32_t rsl = (uint32_t)(tile & (kRSlots - 1));
          if (!mbar_wait(b_rempty + 8 * rsl, ((tile / kRSlots) & 1) ^ 1, g, ST_TIMEOUT_PRODUCER, true, true)) { ok = false; break; }
          mbar_expect_tx(b_rfull + 8 * rsl, kRowFloats * 4);
          bulk_load(sR + rsl * kRowFloats * 4, g.rowsoa + (size_t)(rb + (int)rank) * kRowFloats, kRowFloats * 4,
                    b_rfull + 8 * rsl);
          n_r++;
        }
      }
      // Drain: every copy this CTA issued has landed before the CTA may exit.
      if (item_i > 0) {
        mbar_wait(b_bfull, (item_i - 1) & 1, g, ST_TIMEOUT_DRAIN, false);
        for (uint32_t k = (item_i > 2 ? item_i - 2 : 0); k < item_i; k++)
          mbar_wait(b_cfull + 8 * (k & 1), (k >> 1) & 1, g, ST_TIMEOUT_DRAIN, false);
      }
      for (uint32_t k = (n_r > (uint32_t)kRSlots ? n_r - kRSlots : 0); k < n_r; k++)
        mbar_wait(b_rfull + 8 * (k % kRSlots), (k / kRSlots) & 1, g, ST_TIMEOUT_DRAIN, false);
      const uint32_t ring = (uint32_t)S;
      for (uint32_t k = (n_a > ring ? n_a - ring : 0); k < n_a; k++)
        mbar_wait(b_afull + 8 * (k % ring), (k / ring) & 1, g, ST_TIMEOUT_DRAIN, false);
    }
    __syncwarp();
    role_exit<CTAS>(tmem, false);
    return;
  } else if (warp == 1) {
    // -------------------------------------------------- MMA (CTA 0), relay (CTA 1)
    if (lane == 0) {
      uint32_t tile = 0, item_i = 0;
      uint32_t s = 0, fph = 0;  // ring: stage, parity of the round being consumed
      bool ok = true;
      if (rank == 1) {
        // CTA 1's operands are in place: tell the issuer
        for (int phase = 0; ok && phase < 2; phase++)
        for (ItemCursor cur = first_item<CTAS>(g); ok && cur.it < g.item1; cur.advance(g, n_clusters)) {
          int ct, rb0, rb1;
          if (!cur.part(g, kBN / kBM, kBN, phase, ct, rb0, rb1)) continue;
          if (!mbar_wait(b_bfull, item_i & 1, g, ST_TIMEOUT_MMA)) { ok = false; break; }
          mbar_arrive_cluster(leader_addr(b_bfull));
          item_i++;
          for (int k = (rb1 - rb0 + M - 1) / M * g.nst; k > 0; k--) {
            if (!mbar_wait(b_afull + 8 * s, fph, g, ST_TIMEOUT_MMA)) { ok = false; break; }
            mbar_arrive_cluster(leader_addr(b_afull + 8 * s));
            if (++s == (uint32_t)S) {
              s = 0;
              fph ^= 1;
            }
          }
        }
      } else {
        // This thread's instructions between MMAs are tensor time (an MMA takes 128
        // clocks), so the operand offsets come from a table, one entry ahead.
        const uint32_t a0 = desc_lo(sA), b0 = desc_lo(sB), stage_u = stage_bytes >> 4;
        const int nst = g.nst, n_mma = g.parts * (g.parts + 1) / 2 * g.nb + g.nt;
        for (int phase = 0; ok && phase < 2; phase++)
        for (ItemCursor cur = first_item<CTAS>(g); ok && cur.it < g.item1; cur.advance(g, n_clusters)) {
          int ct, rb0, rb1;
          if (!cur.part(g, kBN / kBM, kBN, phase, ct, rb0, rb1)) continue;
          if (!mbar_wait(b_bfull, item_i & 1, g, ST_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          item_i++;
          for (int rb = rb0; ok && rb < rb1; rb += M, tile++) {
            const uint32_t b = tile & 1;
            if (!mbar_wait(b_acce + 8 * b, ((tile >> 1) & 1) ^ 1, g, ST_TIMEOUT_MMA)) { ok = false; break; }
            const uint32_t d = tmem + b * kBN;
            uint32_t acc = 0;
            int m = 0;
            for (int st = 0; st < nst; st++) {
              if (!mbar_wait(b_afull + 8 * s, fph, g, ST_TIMEOUT_MMA)) { ok = false; break; }
              if (st == 0) tc_fence_after();
              const uint32_t as = a0 + s * stage_u;
              const int m1 = st + 1 == nst ? n_mma : (int)mma_end[st];
              uint2 e = mma_tab[m];
#pragma unroll 2
              while (m < m1) {
                const uint2 cur_e = e;
                e = mma_tab[++m];
                mma_f16<CTAS>(d, as + cur_e.x, b0 + cur_e.y, acc);
                acc = 1;
              }
              // one commit a stage: the accumulator's also frees the tile's last stage
              // (the epilogue passes it on), a second one held the MMAs up 240 clocks
              mma_commit<CTAS>(st + 1 == nst ? b_accf + 8 * b : b_aempty + 8 * s);
              if (++s == (uint32_t)S) {
                s = 0;
                fph ^= 1;
              }
            }
          }
          if (ok) mma_commit<CTAS>(b_bempty);  // the item's B tile is free once these MMAs complete
        }
        // All MMAs this thread issued are complete before TMEM is released and
        // the CTAs exit.
        mma_commit<CTAS>(b_done);
        mbar_wait(b_done, 0, g, ST_TIMEOUT_DRAIN, false);
      }
    }
    __syncwarp();
    role_exit<CTAS>(tmem, true);
    return;
  } else {
    // ---------------------------------------------------------------- epilogue
    const int ew = warp - 2;  // epilogue warp; its TMEM lanes are 32 (warp % 4)..
    const int quarter = warp & 3, part = (ew >> 2) & (4 / SETS - 1), set = SETS == 2 ? ew >> 3 : 0;
    float* fs = scratch + ew * kScratch;
    const uint32_t acce = CTAS == 2 ? leader_addr(b_acce) : b_acce;
    uint32_t tile = 0, item_i = 0, st0 = 0;  // st0: ring stage of the tile's first operands
    const uint32_t back = (uint32_t)(g.nst - 1) % (uint32_t)S;
    bool ok = true;
    // One pass over the CTA's items per phase (ItemCursor::part): the full tiles with
    // the unmasked forms, then the masked tiles, each in a loop of its own.
    auto pass = [&](auto phase_tag) {
    constexpr int kPhase = decltype(phase_tag)::value;
    for (ItemCursor cur = first_item<CTAS>(g); ok && cur.it < g.item1; cur.advance(g, n_clusters)) {
      int ct, rb0, rb1;
      if (!cur.part(g, kBN / kBM, kBN, kPhase, ct, rb0, rb1)) continue;
      const uint32_t cs = item_i & 1;
      if (!warp_wait(b_cfull + 8 * cs, (item_i >> 1) & 1, g, ST_TIMEOUT_EPI)) { ok = false; break; }
      item_i++;
      const float* csl = cslots + cs * kColFloats;
      const float* csw = csl + part * W;
      // centre and half range of a and r over the slab's column groups
      float4 cg = reinterpret_cast<const float4*>(csl + 4 * kBN)[SETS * part];
      if (SETS == 2) {
        const float4 u = cg, v = reinterpret_cast<const float4*>(csl + 4 * kBN)[SETS * part + 1];
        const float lo = fminf(u.x - u.y, v.x - v.y), hi = fmaxf(u.x + u.y, v.x + v.y);
        const float rl = fminf(u.z - u.w, v.z - v.w), rh = fmaxf(u.z + u.w, v.z + v.w);
        const float bad = 0.0f * (u.x + v.x);  // NaN if either group has one
        cg = make_float4(0.5f * (lo + hi) + bad, 0.5f * (hi - lo) * 1.000001f, 0.5f * (rl + rh),
                         0.5f * (rh - rl) * 1.000001f);
      }
      const int q0 = ct * kBN + part * W;
      F2 cacc[CH][2];
#pragma unroll
      for (int c = 0; c < CH; c++) cacc[c][0] = cacc[c][1] = f2(0.0f, 0.0f);
      bool any = false;  // this set had a tile of the item
      for (int rb = rb0; ok && rb < rb1; rb += M, tile++) {
        const uint32_t b = tile & 1;
        const uint32_t last = ring_last(st0, back, S);  // its last stage
        st0 = last + 1 == (uint32_t)S ? 0 : last + 1;
        if (SETS == 2 && (int)b != set) continue;
        any = true;
        const uint32_t rsl = tile & (kRSlots - 1);
        if (!warp_wait(b_rfull + 8 * rsl, (tile / kRSlots) & 1, g, ST_TIMEOUT_EPI)) { ok = false; break; }
        const float* rsp = rslots + rsl * kRowFloats;
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + b * kBN + part * W;
        const int p0 = (rb + (int)rank) * kBM;
        int mode = kPure;
        SlabC sc;
        if constexpr (kPhase == 0 && weighted_num<METRIC>()) {
          mode = slab_mode<METRIC>(*reinterpret_cast<const float4*>(rsp + kRowGrp + 4 * quarter), cg, g.ec, sc);
          if (mode == kPure || mode == kFirst) {
            slab_factors<METRIC>(rsp, csw, sc, fs, g.ec);
            __syncwarp();
          }
        }
        if (!warp_wait(b_accf + 8 * b, (tile >> 1) & 1, g, ST_TIMEOUT_EPI)) { ok = false; break; }
        tc_fence_after();
        float rsum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if constexpr (kPhase == 1 || METRIC == kDebugDot || METRIC == kDebugSum) {
          tile_pairs<METRIC, true, kPhase == 1>(taddr, rsp, csw, cacc, p0, q0, g.ec, rsum);
        } else if (mode == kPure) {
          tile_factor<METRIC, false>(taddr, rsp, csw, sc, fs, cacc, g.ec, p0, q0, rsum);
        } else if constexpr (weighted_num<METRIC>()) {
          if (mode == kFirst) tile_factor<METRIC, true>(taddr, rsp, csw, sc, fs, cacc, g.ec, p0, q0, rsum);
          else if (METRIC == kPearson && mode == kPairFirst)
            tile_pairs<METRIC, false, false>(taddr, rsp, csw, cacc, p0, q0, g.ec, rsum);
          else if (mode == kPairExact)
            tile_pairs<METRIC, true, false>(taddr, rsp, csw, cacc, p0, q0, g.ec, rsum);
        }
        // This warp's reads of the accumulator are complete: the MMA of the tile after the next
        // may overwrite it while the row sums are finished. So are its reads of the row (and,
        // at this set's last tile of the item, the column) parameters, and the MMAs that read
        // the tile's last operands, which a warp passes on. One set of 16 warps gives back two slots
        // of row parameters at a time and takes turns at passing on, for fewer fences: every tile
        // SSIM took 1.2% longer with them and NRMSE 6%, so 1% and 0.5%. Two sets hide a fence a
        // tile (0.5-1%; 2% at 256x256 5x5).
        tc_fence_before();
        __syncwarp();
        const bool pass_on = SETS == 2 ? ew == 8 * set : tile % EW == (uint32_t)ew;
        const bool rows_read = SETS == 2 || b == 1, cols_read = rb + SETS * M >= rb1;
        if (lane == 0) {
          mbar_arrive_tmem(acce + 8 * b);
          if (rows_read || cols_read || pass_on) {
            fence_reads();
            if (rows_read) mbar_arrive_fenced(b_rempty + 8 * rsl);
            if (SETS == 1 && rows_read) mbar_arrive_fenced(b_rempty + 8 * (rsl - 1));
            if (cols_read) mbar_arrive_fenced(b_cempty + 8 * cs);
            if (pass_on) mbar_arrive_fenced(b_aempty + 8 * last);
          }
        }
        // Row sums: 4 lanes per row, then one FP64 atomic add per row and warp (256 a
        // tile, a tenth of the rate the L2 sustains; combining the two halves' warps
        // in shared memory first costs more issue slots than it saves).
        float z = reduce_rows4(rsum);
        const int krow = 2 * (lane & 1) + ((lane >> 1) & 1);
        if (kPhase == 0 && weighted_num<METRIC>() && (mode == kPure || mode == kFirst)) z *= fs[4 * (lane >> 2) + krow];
        const int p = p0 + quarter * 32 + (lane >> 2) + 8 * krow;
        if (p < g.ec.n && !(kPhase == 0 && mode == kZero)) atomicAdd(g.num + p, (double)z);
        __syncwarp();  // (the scratch is rewritten for the next tile)
      }
      if (!ok) break;
      if (!any) {  // (the slot's ranges were read all the same)
        __syncwarp();
        if (lane == 0) {
          fence_reads();
          mbar_arrive_fenced(b_cempty + 8 * cs);
        }
      } else {  // column sums of the item
        float x[4 * CH];
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
          for (int r = 0; r < 2; r++) f2_split(cacc[c][r], x[(c * 2 + r) * 2], x[(c * 2 + r) * 2 + 1]);
        flush_columns<4 * CH>(x, q0, g.ec, g.num);
      }
    }
    };
    pass(std::integral_constant<int, 0>{});
    pass(std::integral_constant<int, 1>{});
    role_exit<CTAS>(tmem, false);
  }
}

// Column parameters of each column tile, permuted so that thread t of an
// epilogue warp finds its four columns of a 16-column chunk (2(t%4) + {0, 1}
// and 8 + 2(t%4) + {0, 1}) in one float4 (col_soa_pos), and the row parameters
// of each 128-row block, in order; each followed by the centre and half range
// of a and r over its four groups (64 columns, 32 rows), which the epilogue's
// slab forms are chosen by. A NaN makes its group's ranges NaN.
// Blocks [0, n_ctp): column tiles; [n_ctp, n_ctp + n_rbp): row blocks.
__global__ void k_sym_soa(const BlockParams* __restrict__ params, int n_ctp, float* __restrict__ colsoa,
                          float* __restrict__ rowsoa) {
  const int i = threadIdx.x;
  __shared__ float4 wm[8];
  const bool col = blockIdx.x < n_ctp;
  const int width = col ? kBN : kBM;
  const int tile = col ? blockIdx.x : blockIdx.x - n_ctp;
  float* o = col ? colsoa + (size_t)tile * kColFloats : rowsoa + (size_t)tile * kRowSoaFloats;
  if (i < width) {
    const BlockParams p = params[(size_t)tile * width + i];
    const int pos = col ? col_soa_pos(i) : i;
    o[pos] = p.a;
    o[width + pos] = p.r;
    o[2 * width + pos] = p.sigma;
    o[3 * width + pos] = p.mu;
    float4 m = make_float4(p.a, p.a, p.r, p.r);
    const bool bad = !(p.a - p.a == 0.0f) || !(p.r - p.r == 0.0f);
    for (int s = 16; s; s >>= 1) {
      m.x = fminf(m.x, __shfl_xor_sync(0xffffffffu, m.x, s));
      m.y = fmaxf(m.y, __shfl_xor_sync(0xffffffffu, m.y, s));
      m.z = fminf(m.z, __shfl_xor_sync(0xffffffffu, m.z, s));
      m.w = fmaxf(m.w, __shfl_xor_sync(0xffffffffu, m.w, s));
    }
    if (__any_sync(0xffffffffu, bad)) m = make_float4(nanf(""), nanf(""), nanf(""), nanf(""));
    if ((i & 31) == 0) wm[i >> 5] = m;
  }
  __syncthreads();
  if (i < 4) {
    const int per = width / 128;  // warps per group
    float4 m = wm[i * per];
    if (per == 2) {
      const float4 b = wm[i * per + 1];
      const bool bad = m.x != m.x || b.x != b.x;
      m = make_float4(fminf(m.x, b.x), fmaxf(m.y, b.y), fminf(m.z, b.z), fmaxf(m.w, b.w));
      if (bad) m.x = m.y = m.z = m.w = nanf("");
    }
    // half ranges rounded up, so that they bound the distance to the rounded centre
    const float ca = 0.5f * (m.x + m.y), cr = 0.5f * (m.z + m.w);
    reinterpret_cast<float4*>(o + 4 * width)[i] =
        make_float4(ca, fmaxf(m.y - ca, ca - m.x) * 1.0000002f, cr, fmaxf(m.w - cr, cr - m.z) * 1.0000002f);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// U as [chunk][row][64 columns] (128-byte rows, SWIZZLE_128B), boxes of
// box_rows rows of sc chunks. Where the pitch ends half way through the last chunk, its other half
// reads the next row's first columns, which no MMA uses (the buffer has 64 bytes
// past the last row).
bool make_map(CUtensorMap* m, const __half* ptr, int pitch, int rows, int sc, int box_rows) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)kChunk, (cuuint64_t)rows, (cuuint64_t)((pitch + kChunk - 1) / kChunk)};
  cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)kChunk * 2};
  cuuint32_t box[3] = {(cuuint32_t)kChunk, (cuuint32_t)box_rows, (cuuint32_t)sc};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

constexpr size_t kFixedSmem =
    (2 * (size_t)kColFloats + kRSlots * kRowFloats + (size_t)kEpiWarps * kScratch) * 4 + kBarBytes + kTabBytes;

}  // namespace

// Shape for K ellipse pixels: CTAs per tile, and a ring of stages of whole
// row-block tiles (three or more) or of single chunks (three or more).
bool plan_shape(int K, int ctas, bool whole, TcPlan* p) {
  if (K <= 0) return false;
  const SplitLayout l = split_layout(K);
  const int nch = (l.pitch + kChunk - 1) / kChunk;
  const int cols = nch * (kBN / kBM / ctas);  // chunks of 128 rows of the column tile in a CTA
  const int chunks = (int)((kMaxSmem - kFixedSmem) / kChunkBytes) - cols;  // of the ring
  const int sc = whole ? nch : 1;
  if (chunks < 3 * sc) return false;
  const int st = std::min(kMaxStages, chunks / sc);
  *p = TcPlan{ctas, sc, st, kFixedSmem + (size_t)(cols + st * sc) * kChunkBytes};
  return true;
}

bool plan_gram_tc(int K, TcPlan* p) {
  return plan_shape(K, 1, true, p) || plan_shape(K, 2, true, p) || plan_shape(K, 2, false, p);
}

// The shape a table entry names: whole-tile stages (tr 1) or single chunks.
bool plan_choice(int K, const TcChoice& c, TcPlan* p) {
  return c.tr ? plan_shape(K, 1, true, p) || plan_shape(K, 2, true, p) : plan_shape(K, 2, false, p);
}

int gram_tc_candidates(int K, TcChoice* out, int cap) {
  int n = 0;
  TcPlan p;
  for (int tr : {1, 0})
    if (plan_choice(K, TcChoice{kBN, tr, 128}, &p))
      for (int L : {128, 32, 16, 8, 4})
        if (n < cap) out[n++] = TcChoice{kBN, tr, L};
  return n;
}

bool gram_tc_valid(int K, const TcChoice& c) {
  TcPlan p;
  const bool L = c.L == 128 || c.L == 32 || c.L == 16 || c.L == 8 || c.L == 4;
  return L && (c.bn == 256 || c.bn == 128) && (c.tr == 0 || c.tr == 1) && plan_choice(K, c, &p);
}

size_t gram_tc_soa_floats(int n_pad) {
  return (size_t)(n_pad / kBN) * kColFloats + (size_t)(n_pad / kBM) * kRowSoaFloats;
}

long long gram_tc_items(int n, int bn, int* L_out, int num_sms, int max_L) {
  const int m = bn / kBM;
  const int n_rb = (n + kBM - 1) / kBM, n_ct = (n + bn - 1) / bn;
  auto items = [&](int L) {
    const int runs = (n_rb + L - 1) / L;
    return items_before_run(runs, n_ct, L / m);
  };
  int L = max_L > 0 && max_L < kMaxRun ? max_L : kMaxRun;
  while (L > 2 && items(L) < 16LL * num_sms) L >>= 1;
  if (L < m) L = m;
  if (L_out) *L_out = L;
  return items(L);
}

cudaError_t launch_gram_tc(const __half* U, int K, int n_pad, const BlockParams* params, float* soa_ws, EpiConsts ec,
                           double* num, int num_sms, int* status, cudaStream_t st, int shard, int n_shards,
                           const TcDebug* dbg, const TcChoice* choice) {
  TcPlan plan;
  const bool planned = (choice && choice->bn && plan_choice(K, *choice, &plan)) || plan_gram_tc(K, &plan);
  if (!planned || n_pad % kBN != 0 || n_shards < 1 || shard < 0 || shard >= n_shards) return cudaErrorInvalidValue;
  if (ec.n <= 0) return cudaSuccess;
  const SplitLayout l = split_layout(K);
  TcArgs g;
  g.parts = l.parts;
  g.nb = l.nb;
  g.nt = l.nt;
  g.nch = (l.pitch + kChunk - 1) / kChunk;
  g.sc = plan.sc;
  g.nst = (g.nch + plan.sc - 1) / plan.sc;
  g.stages = plan.stages;
  g.n_rb = (ec.n + kBM - 1) / kBM;
  g.n_ct = (ec.n + kBN - 1) / kBN;
  int L;
  const long long items = gram_tc_items(ec.n, kBN, &L, num_sms, choice ? choice->L : 0);
  g.L = L;
  g.h = L / (kBN / kBM);
  g.n_runs = (g.n_rb + L - 1) / L;
  // panels of column tiles whose operands fill at most 48 MB of L2
  g.panel = std::max(1, (int)(((size_t)48 << 20) / ((size_t)kBN * l.pitch * 2)));
  g.n_panels = (g.n_ct + g.panel - 1) / g.panel;
  g.item0 = items * shard / n_shards;
  g.item1 = items * (shard + 1) / n_shards;
  const int n_ctp = n_pad / kBN, n_rbp = n_pad / kBM;
  float* colsoa = soa_ws;
  float* rowsoa = soa_ws + (size_t)n_ctp * kColFloats;
  g.colsoa = colsoa;
  g.rowsoa = rowsoa;
  g.ec = ec;
  g.num = num;
  g.status = status;
  g.timeout_ns = dbg && dbg->timeout_ns ? dbg->timeout_ns : 4000000000ull;
  g.withhold = dbg ? dbg->withhold_tile : -1;
  k_sym_soa<<<n_ctp + n_rbp, 256, 0, st>>>(params, n_ctp, colsoa, rowsoa);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (g.item0 >= g.item1) return cudaSuccess;
  CUtensorMap mU, mB;
  if (!make_map(&mU, U, l.pitch, n_pad, plan.sc, kBM) || !make_map(&mB, U, l.pitch, n_pad, plan.sc, kBN / plan.ctas))
    return cudaErrorInvalidValue;
  const int smem = (int)plan.smem;
  // one CTA per SM: as many CTAs or pairs of CTAs as can be resident at once
  auto launch = [&](auto kern) -> cudaError_t {
    // (the same value in every call: another thread's launch may lie between)
    cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    if (r != cudaSuccess) return r;
    int groups = num_sms;
    if (plan.ctas == 2) {
      static std::atomic<int> resident[16];  // pairs per device, whatever the ring
      int dev = 0;
      if ((r = cudaGetDevice(&dev)) != cudaSuccess) return r;
      groups = dev < 16 ? resident[dev].load() : 0;
      if (groups == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * std::max(1, num_sms / 2));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        r = cudaOccupancyMaxActiveClusters(&groups, kern, &cfg);
        if (r != cudaSuccess) return r;
        groups = std::max(1, std::min(groups, num_sms / 2));
        if (dev < 16) resident[dev].store(groups);
      }
    }
    const int grid = plan.ctas * (int)std::min<long long>(g.item1 - g.item0, groups);
    kern<<<grid, kThreads, smem, st>>>(mU, mB, g);
    return cudaGetLastError();
  };
#define SRED_TC(M) return plan.ctas == 2 ? launch(k_gram_tc<M, 2>) : launch(k_gram_tc<M, 1>)
  switch (ec.metric) {
    case kPearson: SRED_TC(kPearson);
    case kSsim: SRED_TC(kSsim);
    case kNrmse: SRED_TC(kNrmse);
    case kNrmseW: SRED_TC(kNrmseW);
    case kDebugDot: SRED_TC(kDebugDot);
    case kDebugSum: SRED_TC(kDebugSum);
    default: return cudaErrorInvalidValue;
  }
#undef SRED_TC
}

}  // namespace sred
