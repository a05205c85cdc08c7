// Initial k-NN over leaf blocks on the 5th-generation tensor cores (tcgen05),
// for EUCLIDEAN and COSINE: the mixed-precision leaf stage.
//
// Also the filter in front of the FP32 leaf stage (BOUND, leaf_stage_filtered below).
//
// Same blocks and same union-over-trees rule as the FP32 leaf stage (which
// replaces findInitialStateOfAproximated*KNN, euclideandistancematrixgpu.cu:107-1031),
// but every (query, candidate) key of a block comes from one BF16 GEMM tile:
//     key ~= |x|^2 + |y|^2 - 2 x.y      (EUCLIDEAN, norms of the BF16 rows)
//     key ~= 1 - x.y                     (COSINE, rows normalised before rounding)
// with FP32 accumulation in tensor memory.  Each point keeps its best kq (2k,
// at most 32) approximate candidates over all trees; k_rerank then recomputes
// those kq keys exactly in FP32 (the reference's order) and keeps the best k.
// When the BF16 products and FP32 sums are exact (integer data below 2^8 per
// coordinate and 2^24 per sum, e.g. the integer-mixture workload) the result
// equals the FP32 leaf stage bit for bit.
//
// Per tree the 16-bit rows are first copied into the tree's order
// (k_permute_operand), so that a block's candidate tiles are plain 2-D boxes.
// One thread block per (leaf, QT x 128 queries), warp-specialised:
//   * a producer thread streams the block's candidates with TMA: boxes of 64
//     rows x 64 elements (128-byte swizzle, 8 KB) into a ring;
//   * an MMA thread issues tcgen05.mma.cta_group::1.kind::f16, M=128 N=64 K=16:
//     the queries (A) stay in tensor memory for the whole block, the candidates
//     (B) come from the ring, and QT query tiles share each candidate box; the
//     FP32 accumulators rotate over NB 64-column buffers per query tile (one up to
//     128 dims, where a tile's products wait for the last tile's to be read; two above);
//   * four epilogue warps per query tile, one per lane quarter: a thread owns a
//     query row.  It reads a tile's two 32-column slices with tcgen05.ld
//     32x32b.x32, filters the products against the row's bound into survivor
//     bits, and appends the few survivors (product, column) to the row's buffer
//     in an L2-resident scratch.
// The stages meet only at mbarriers, so loads, products and filters of different
// tiles overlap; no barrier spans the block between its prologue and end.
// k_leaf_tc_merge then sorts each row's survivors and merges them into its list.
//
// What bounds it, and why this split.  The products of a 128 x 128 x 128 tile
// take ~710 cycles of an SM's tensor pipe at the measured bf16 rate; the filter
// needs two FP32 pipe and two ALU pipe cycles per 32 keys and scheduler, ~260-320
// cycles.  Merging inside the tile kernel (a warp per survivor, two block barriers
// per tile) held both to a few percent: 16 warps' latencies, and every warp waiting
// for the slowest.  So the tile kernel only filters (16 epilogue warps per SM: two
// blocks of two query tiles), and sorting runs at full occupancy in a kernel of
// its own.  Integer mixture, 1M x 128, 8 trees, leaf 2048, k=16, tiles of all
// trees: 30.8 ms with the in-kernel merge, 12.7 ms in this form (of which the merge
// kernel 2.2 ms); 10M x 96 FP16 COSINE, 15 trees, leaf 4096: 431 -> 182 ms.  What
// is left is the epilogue's latency chain (issue slots 50 % busy, tensor pipe
// 28 % in the first tree).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "knn_internal.cuh"
#include "knn_kernels.cuh"

namespace knn {

namespace {
constexpr int kBM = 128;              // query rows of one accumulator
constexpr int kTN = 64;               // candidate columns of one tile
constexpr int kKC = 64;               // 16-bit elements per 128-byte swizzled row
constexpr int kBoxBytes = kTN * 128;  // one 64 x 64 candidate box
constexpr int kRing = 4;              // candidate boxes in flight (at least a tile's, four)
// Survivors a row's buffer holds: rows of a later tree whose list is still poor
// may see a hundred; 320 or 512 measured no faster (longer scratch rows).
constexpr int kCap = 192;
constexpr int kFlushAt = kCap - kTN;  // a fuller buffer could not take another tile
constexpr int kFlushMin = 24;         // rows merged along when one row's buffer is full
// Rows (of whole blocks) per launch: bounds the survivor scratch, 1.5 KB a row, at 805 MB.  Half as
// many cost 6 % of the headline build (22.7 -> 24.0 ms) and 5 % at 10M rows, a quarter 14 %: each
// launch ends in a tail.  Less is used where memory is short.
constexpr int64_t kChunkRows = 1 << 19;
constexpr uint32_t kOverflow = 0xFFFFFFFFu;  // FP32 filter: more survivors than the buffer holds, evaluate the block
constexpr uint32_t kListed = 0x80000000u;  // count flag (first tree): the row's list was already written
constexpr int kBand = 1024;           // block columns covered by the listed-column bitmap at a time
constexpr int kBandWords = kBand / 32 + 1;
constexpr int kNormSlots = 8;         // tiles of candidate norms staged ahead
constexpr int kMergeRows = 4;         // rows merged together by a warp (independent chains)
constexpr int kInsertMax = 5;         // candidates up to which one-by-one insertion beats sort and merge
constexpr int kBoundRows = 4;         // the same for the bounding pass's selection
constexpr float kSlack = 4.76837158203125e-07f;  // 2^-21: filter widening, eight units of FP32 rounding
// Bounding pass: in the first kPrepassTrees trees, blocks of at least
// kPrepassMin columns run their tiles once more beforehand; the group minima
// (kGroups 32-column slices per row, wrapping, row stride kGS) overlay the
// epilogue warp's shared memory.  In the second tree it replaces the tails of
// rows whose first leaf was poor, which alone cost more than the pass: integer
// mixture as above, tiles 14.9 -> 12.7 ms; a third tree's pass gains nothing.
constexpr int kPrepassTrees = 2;
constexpr int kPrepassMin = 256;
constexpr int kGroups = 64;
constexpr int kGS = kGroups + 1;
// Shared memory of one epilogue warp: a slice's products and the bitmaps of
// listed columns (in the bounding pass: the group minima).
constexpr int kDumpStride = 144;  // bytes of one row's 32 products, padded: 16-byte stores hit distinct banks
constexpr int kWarpDump = 32 * kDumpStride;
constexpr int kWarpBits = 32 * kBandWords * 4;
constexpr int kWarpBytes = kWarpDump + kWarpBits;
constexpr int kNormBytes = kNormSlots * (kTN + 4) * 4;  // -|y|^2 of a tile's columns, then the largest |y|^2
static_assert(kWarpBytes >= 32 * kGS * 4, "group minima fit");
static_assert(kWarpBytes % 16 == 0, "16-byte accesses");

// Instruction descriptor of kind::f16: D f32 (bits 4-5 = 1), A and B format
// at 7-9 and 10-12 (0 f16, 1 bf16; A and B always the same type), A and B
// K-major (15, 16 = 0), N>>3 at 17-22, M>>4 at 24-28.
constexpr uint32_t idesc_for(bool f16) {
  return (1u << 4) | ((f16 ? 0u : 1u) << 7) | ((f16 ? 0u : 1u) << 10) | ((uint32_t)(kTN >> 3) << 17) |
         ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: start address
// (>>4) in bits 0-13, leading offset 1 (unused for swizzled K-major) at 16-29,
// stride 1024 B (>>4 = 64) between 8-row atoms at 32-45, version 1 at 46-47,
// base offset 0, layout type 2 (SWIZZLE_128B) at 61-63.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)64 << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// Phase completion; may suspend the thread for at most about kPollNs.
constexpr uint32_t kPollNs = 2000;
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kPollNs)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity; false once kWaitNs of wall time
// (globaltimer) have passed, or once another wait of the block has given up.
// The first to give up records it in the block's status and the error words:
// err[0] stops the build's later blocks, err[1] stays until the host reports it.
// (FP32 filter: words of the build's own, no failure; the block hands its tree to dense tiles.)
constexpr uint64_t kWaitNs = 20ull * 1000 * 1000;  // 20 ms; a tile takes under a microsecond
constexpr uint32_t kSpinLimit = 1u << 20;
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* status, int* err) {
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < kSpinLimit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*status != 0) return false;
    if (global_ns() - t0 > kWaitNs) break;
  }
  // the time may have passed between the last poll and the clock (a time-sliced GPU)
  if (mbar_try_wait(bar, parity)) return true;
  *status = 1;
  atomicExch(err, 1);
  atomicOr(err + 1, 1);
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* status, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, status, err);
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(p));
  return p != 0;
}

// D (tensor memory) += A (tensor memory) x B (shared memory descriptor)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tma_load_box(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
          "r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// Issue only: the values are valid after tmem_wait_ld().
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
// The loaded registers pass through the wait, so that no use of them can be
// scheduled ahead of it.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(v[i]));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]),
      "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
      "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}

// Two FP32 lanes in one instruction (each lane rounded as the scalar form).
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// ------------------------------------------------------------- list merge --
// Lists and candidates are (ordered key, id) pairs compared as one 64-bit
// number: ordered keys are the FP32 keys mapped to integers of the same order.
constexpr uint32_t kNoKey = 0xFFFFFFFFu;
__device__ __forceinline__ float from_orderable(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o ^ 0x80000000u) : ~o);
}
__device__ __forceinline__ bool pair_less(uint32_t ak, uint32_t ai, uint32_t bk, uint32_t bi) {
  return (((uint64_t)ak << 32) | ai) < (((uint64_t)bk << 32) | bi);
}

// One compare-exchange step of R interleaved networks: lanes with keep_small
// keep the smaller pair of themselves and lane ^ m.
template <int R>
__device__ __forceinline__ void exchange_rows(uint32_t (&k)[R], uint32_t (&id)[R], int m, bool keep_small) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint32_t ok = __shfl_xor_sync(0xFFFFFFFFu, k[i], m);
    const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, id[i], m);
    if (pair_less(ok, oi, k[i], id[i]) == keep_small) {
      k[i] = ok;
      id[i] = oi;
    }
  }
}
// Equal pairs (two empty entries) may be exchanged either way: both are the same.

// Ascending sort of the first `cnt` lanes (the others empty) of R rows: the
// levels of the bitonic network up to the power of two that holds cnt.  The
// steps are a loop: R rows keep the pipes busy, and straight-line code would not
// stay in the instruction cache between merges.
template <int R>
__device__ __forceinline__ void sort_rows(uint32_t (&k)[R], uint32_t (&id)[R], int cnt) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int size = 2; size <= 32 && (size >> 1) < cnt; size <<= 1) {  // warp-uniform
#pragma unroll 1
    for (int m = size >> 1; m >= 1; m >>= 1)
      exchange_rows<R>(k, id, m, ((lane & size) == 0) == ((lane & m) == 0));
  }
}

// The candidates of the first `cnt` lanes one by one into R sorted lists: the
// lanes whose entry is greater form a suffix, which shifts up one lane (the last
// entry drops out).  An empty candidate is greater than every entry.
template <int R>
__device__ __forceinline__ void insert_rows(uint32_t (&lk)[R], uint32_t (&li)[R], const uint32_t (&ck)[R],
                                            const uint32_t (&ci)[R], int cnt) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int e = 0; e < cnt; ++e) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint32_t k1 = __shfl_sync(0xFFFFFFFFu, ck[i], e), i1 = __shfl_sync(0xFFFFFFFFu, ci[i], e);
      const uint32_t uk = __shfl_up_sync(0xFFFFFFFFu, lk[i], 1), ui = __shfl_up_sync(0xFFFFFFFFu, li[i], 1);
      const bool after = pair_less(k1, i1, lk[i], li[i]);
      const bool before = lane == 0 || !pair_less(k1, i1, uk, ui);  // the entry below stays
      if (after) {
        lk[i] = before ? k1 : uk;
        li[i] = before ? i1 : ui;
      }
    }
  }
}

// Lists <- the 32 smallest of list and sorted candidates.
template <int R>
__device__ __forceinline__ void merge_lower_rows(uint32_t (&lk)[R], uint32_t (&li)[R], const uint32_t (&ck)[R],
                                                 const uint32_t (&ci)[R]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint32_t rk = __shfl_sync(0xFFFFFFFFu, ck[i], 31 - lane);
    const uint32_t ri = __shfl_sync(0xFFFFFFFFu, ci[i], 31 - lane);
    if (pair_less(rk, ri, lk[i], li[i])) {  // min(list, reversed candidates) is bitonic
      lk[i] = rk;
      li[i] = ri;
    }
  }
#pragma unroll 1
  for (int m = 16; m >= 1; m >>= 1) exchange_rows<R>(lk, li, m, (lane & m) == 0);
}

// Tensor-memory columns of a block: QT * NB accumulators, then QT query tiles.
// Up to 128 dims a block takes 128 columns per query tile, else 256.
template <int NCH, int QT>
struct TmemPlan {
  static constexpr int kTotal = NCH <= 2 ? 128 * QT : 256;
  static constexpr int kA = NCH * 32;                              // columns of one query tile
  static constexpr int kNB = (kTotal - QT * kA) / (QT * kTN);      // accumulators per query tile
  static constexpr int kA0 = QT * kNB * kTN;
  static constexpr int kBlocks = NCH <= 2 && QT == 1 ? 3 : 2;      // resident blocks per SM
  static_assert(kNB >= 1 && kA0 + QT * kA <= kTotal && kBlocks * kTotal <= 512, "tensor memory plan");
};

}  // namespace

struct LeafTcArgs {
  const uint16_t* Xp;     // [n][ldr] 16-bit rows in the tree's order
  const float* np;        // [n] their norms in the tree's order (EUCLIDEAN)
  const int32_t* perm;    // [n] the tree's order
  const int32_t* plist;   // [n][kq] later trees: the position of every list entry, rows in the tree's order
  const int64_t* ftab;    // leaf table (reference-rule trees) or null
  SegView segs;
  uint32_t* akey;         // [n][kq] ordered keys
  uint32_t* aid;          // [n][kq]
  // [blocks of the launch][128 QT][kCap] survivors: product (FP32 filter: unset, then the ordered exact key),
  // block column (then the id)
  uint2* surv;
  // FP32 filter (BOUND)
  const float* X;         // [n][dpad] FP32 rows
  const float* norms;     // [n] FP32 norms (COSINE)
  const float* dp;        // [n] bounds of the 16-bit rows' errors, in the tree's order
  const float* rkey;      // [n][k] lists: exact keys
  const unsigned int* maxabs;
  unsigned long long* pair_counter;
  unsigned long long* survivors;  // FP32 filter: [-1] of the tree before, [0] of this tree
  unsigned long long survivor_limit;
  bool give_up;           // test hook: every block behaves as if a wait had given up
  float g, g1;            // FP32 rounding of a key; of a tile's sums
  int d, dpad, metric;
  uint32_t* count;        // [blocks of the launch][128 QT] survivors of each row, kListed
  int64_t block0;         // first block of the launch
  int* err;
  int64_t n;
  uint32_t idesc;
  int ldr, ksteps;        // row stride in elements; 16-element steps holding dims
  int k, kq, qtiles, glog;
};

// FP32 filter.  The 16-bit rows are s * (x - c) (COSINE: of the unit rows), c a
// member row of the leaf, so that rounding errors scale with the leaf and not with
// the data's offset; s is the power of two that brings the largest |x| of all
// rows into [2^13, 2^14), so differences stay inside the FP16 range.
__device__ __forceinline__ float bound_scale(const LeafTcArgs& a) {
  if (a.metric == KNN_METRIC_COSINE) return 8192.f;
  const float m = __uint_as_float(*a.maxabs);
  if (!(m > 0.f && m < __int_as_float(0x7F800000))) return 1.f;
  int e;
  frexpf(m, &e);  // m in [2^(e-1), 2^e)
  return ldexpf(1.f, max(-126, min(126, 14 - e)));
}
// A scaled distance that neither the pair of an exact key reaches nor any pair
// with a smaller key.  Slack for what a key may lose to underflow of its squares
// (EUCLIDEAN, d 2^-138), or for its rounding (COSINE: |u - v|^2 = 2 key, and the
// dot product, both norms and the division round by less than 1.5 g in all).
__device__ __forceinline__ float key_distance(float key, float scale, const LeafTcArgs& a) {
  const float q = a.metric == KNN_METRIC_COSINE ? 2.f * fmaxf(key, 0.f) + 3.f * a.g : key + (float)a.d * 2.8698593e-42f;
  return scale * __fsqrt_rn(q) * (1.f + a.g);
}
// The same for pairs of which only the 16-bit rows' squared distance (at most
// sq) and error bounds are known.  Distances whose key overflows bound nothing.
__device__ __forceinline__ float minimum_distance(float sq, float err, float scale, const LeafTcArgs& a) {
  const float r = __fsqrt_rn(fmaxf(sq, 0.f)) + err;
  const float slack = a.metric == KNN_METRIC_COSINE ? 6.f * a.g : (float)a.d * 5.7397186e-42f;
  const float t = __fsqrt_rn(r * r + scale * (scale * slack)) * (1.f + 2.f * a.g);
  return t < scale * 1.8e19f ? t : __int_as_float(0x7F800000);
}

// FP32 filter: whether dense tiles take the tree instead, by the survivors that
// the tile kernel counted (tree: this one's; else the one before, whose answer
// this one inherits).
__device__ __forceinline__ bool too_many(const LeafTcArgs& a, int tree) {
  return *reinterpret_cast<volatile unsigned long long*>(a.survivors + tree) > a.survivor_limit;
}

// Block b's leaf rows [lo, hi), candidate block [blo, bhi) (positions in the
// tree's order) and first query row q0 of the leaf.
struct BlockRange {
  int64_t lo, hi, blo, bhi, j;
  SegEntry seg;
  int q0;
};
template <int QT>
__device__ __forceinline__ BlockRange block_range(const LeafTcArgs& a, int64_t b) {
  BlockRange g{};
  const int64_t leaf = b / a.qtiles;
  g.q0 = (int)(b - leaf * a.qtiles) * (kBM * QT);
  if (a.ftab) {  // explicit leaf table (reference-rule trees)
    const int64_t* e = a.ftab + 4 * leaf;
    g.lo = e[0];
    g.hi = e[1];
    g.blo = e[2];
    g.bhi = e[3];
  } else if (a.glog == 0) {
    g.seg = a.segs.leaf(leaf, &g.j);
    leaf_block(g.seg, g.j, a.k, &g.lo, &g.hi, &g.blo, &g.bhi);
  } else {
    // 2^glog sibling leaves, each its own block (the host checks that every
    // leaf holds k+1 points), as one tile: a row keeps only its own leaf's
    // columns
    g.seg = a.segs.leaf(leaf << a.glog, &g.j);
    g.lo = g.blo = g.seg.off + node_lo(g.seg.n, g.seg.depth, g.j);
    g.hi = g.bhi = g.seg.off + node_lo(g.seg.n, g.seg.depth, g.j + (int64_t(1) << a.glog));
  }
  return g;
}

// Merge the buffered survivors of the rows in `rows` (warp-uniform) into their
// lists, kMergeRows rows at a time: every row's loads, sort and merge are
// independent chains.  Lane r holds row r's id, norm, count and bound; surv the
// rows' buffers (product, block column); np and perm start at the block.  Returns the
// bounds, lowered to the new list tails.  EXACT: the buffers hold ordered exact
// keys and ids, the lists FP32 keys (+inf without id: empty).
template <int METRIC, bool EXACT = false>
__device__ __forceinline__ float merge_survivors(uint32_t* akey, uint32_t* aid, const float* np, const int32_t* perm,
                                                 int kq, const uint2* surv, int qid, float myn, int cnt, float tk,
                                                 uint32_t have, uint32_t rows) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  while (rows) {
    uint32_t lk[kMergeRows], li[kMergeRows], ck[kMergeRows], ci[kMergeRows];
    int r[kMergeRows], c[kMergeRows];
    int most = 0;
    bool fresh = true;  // warp-uniform
#pragma unroll
    for (int i = 0; i < kMergeRows; ++i) {  // fewer rows left: the last one again (same result)
      r[i] = rows ? __ffs(rows) - 1 : r[i > 0 ? i - 1 : 0];
      rows &= rows - 1;
    }
#pragma unroll
    for (int i = 0; i < kMergeRows; ++i) {
      const int id = __shfl_sync(0xFFFFFFFFu, qid, r[i]);
      c[i] = __shfl_sync(0xFFFFFFFFu, cnt, r[i]);
      most = max(most, c[i]);
      lk[i] = kNoKey;
      li[i] = kNoId;
      fresh = fresh && !((have >> r[i]) & 1u);
      if (lane < kq && ((have >> r[i]) & 1u)) {
        lk[i] = akey[(size_t)id * kq + lane];
        li[i] = aid[(size_t)id * kq + lane];
        if (EXACT) lk[i] = li[i] == kNoId ? kNoKey : orderable(__uint_as_float(lk[i]));
      }
    }
    for (int e0 = 0; e0 < most; e0 += 32) {
#pragma unroll
      for (int i = 0; i < kMergeRows; ++i) {
        const float xn = __shfl_sync(0xFFFFFFFFu, myn, r[i]);
        ck[i] = kNoKey;
        ci[i] = kNoId;
        if (e0 + lane < c[i]) {
          const uint2 v = surv[r[i] * kCap + e0 + lane];
          if (EXACT) {
            ck[i] = v.x;
            ci[i] = v.y;
            continue;
          }
          const float dot = __uint_as_float(v.x);
          const uint32_t p = v.y;
          ck[i] = orderable(METRIC == KNN_METRIC_EUCLIDEAN ? __fmaf_rn(-2.f, dot, __fadd_rn(xn, np[p]))
                                                           : __fsub_rn(1.f, dot));
          ci[i] = (uint32_t)perm[p];
        }
      }
      if (most - e0 <= kInsertMax) {
        insert_rows<kMergeRows>(lk, li, ck, ci, most - e0);
        continue;
      }
      sort_rows<kMergeRows>(ck, ci, most - e0);
      if (fresh && e0 == 0) {  // empty lists: the sorted candidates are the lists
#pragma unroll
        for (int i = 0; i < kMergeRows; ++i) {
          lk[i] = ck[i];
          li[i] = ci[i];
        }
      } else {
        merge_lower_rows<kMergeRows>(lk, li, ck, ci);
      }
    }
#pragma unroll
    for (int i = 0; i < kMergeRows; ++i) {
      const int id = __shfl_sync(0xFFFFFFFFu, qid, r[i]);
      if (lane < kq) {
        akey[(size_t)id * kq + lane] =
            !EXACT ? lk[i] : li[i] == kNoId ? 0x7F800000u : __float_as_uint(from_orderable(lk[i]));
        aid[(size_t)id * kq + lane] = li[i];
      }
      const float tail = from_orderable(__shfl_sync(0xFFFFFFFFu, lk[i], kq - 1));
      if (lane == r[i] && tail < tk) tk = tail;  // NaN: an empty slot
    }
  }
  __syncwarp();
  return tk;
}

// One block per (leaf, QT x 128 queries).  FIRST: the launch of the first
// tree, whose lists start empty and are all written.  PRE: blocks of
// kPrepassMin columns or more run their tiles twice: pass 0 records each row's
// smallest key' (below) in each of kGroups column groups; the kq-th smallest
// group minimum belongs to kq distinct candidates, so, widened by the rounding
// of key' against the exact key, it bounds the kq-th key of the list after this
// tree, and pass 1 filters against it from its first tile on.
// Later trees: the block's columns that hold an id already in a row's list
// (k_list_positions) are kept as a bitmap, kBand columns at a time, and masked
// out of the survivors, so a candidate meets a list at most once and merging
// needs no duplicate check.
// Row filter, a superset of what the exact rule (key <= the row's list tail
// tk) can admit: key' = |y|^2 - 2 x.y (EUCLIDEAN) or -x.y (COSINE) against
// thr = tk - |x|^2 (or tk - 1) widened by 2^-21 (|tk| + |x|^2 + max|y|^2),
// which bounds the rounding of both the key and the threshold.  A tail from an
// earlier tile is looser than the current one, never tighter.  Every
// survivor's exact key is computed at its merge and ranked there.
template <int METRIC, bool BOUND, bool FIRST, bool PRE, int NCH, int QT>
__global__ void __launch_bounds__(64 + 128 * QT, TmemPlan<NCH, QT>::kBlocks)
    k_leaf_tc(const __grid_constant__ CUtensorMap bmap, const __grid_constant__ LeafTcArgs a) {
  using Plan = TmemPlan<NCH, QT>;
  constexpr int NB = Plan::kNB, RING = kRing;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* ring = smem;
  unsigned char* warp_area = ring + RING * kBoxBytes;
  float* tnorms = reinterpret_cast<float*>(warp_area + 4 * QT * kWarpBytes);  // [kNormSlots][kTN + 4]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(tnorms) + kNormBytes);
  // ring full [RING], ring empty [RING], accumulators full [QT][NB], empty [QT][NB], norms full, empty, drained
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * RING;
  const uint32_t bar_afull = bar_empty + 8 * RING, bar_aempty = bar_afull + 8 * QT * NB;
  const uint32_t bar_nfull = bar_aempty + 8 * QT * NB, bar_nempty = bar_nfull + 8 * kNormSlots;
  const uint32_t bar_done = bar_nempty + 8 * kNormSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * RING + 2 * QT * NB + 2 * kNormSlots + 1);
  int* status_p = reinterpret_cast<int*>(tmem_slot + 1);
  volatile int* status = status_p;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);  // warp-uniform
  const BlockRange range = block_range<QT>(a, a.block0 + blockIdx.x);
  const int64_t lo = range.lo, blo = range.blo, bhi = range.bhi;
  const int nq = (int)(range.hi - lo), q0 = range.q0;
  if (q0 >= nq) return;  // whole block, before any barrier or allocation
  const int nb = (int)(bhi - blo);
  const int qts = min(QT, (nq - q0 + kBM - 1) / kBM);  // query tiles with rows
  const int nt = (nb + kTN - 1) / kTN;
  // columns per group of the bounding pass, and its tiles: enough groups for the kq-th minimum
  const int gw = nb <= 8 * kGroups ? 8 : nb <= 16 * kGroups ? 16 : 32;
  const int npre = PRE && nb >= kPrepassMin && nb >= gw * (a.kq + a.kq / 4) && a.glog == 0 ? nt : 0;
  const int nsteps = npre + nt;

  if (warp == 4 * QT) {  // producer warp: barriers
    if (lane == 0) {
      for (int i = 0; i < RING; ++i) {
        mbar_init(bar_full + 8 * i, 1);
        mbar_init(bar_empty + 8 * i, 1);
      }
      for (int i = 0; i < QT * NB; ++i) {
        mbar_init(bar_afull + 8 * i, 1);
        mbar_init(bar_aempty + 8 * i, 4);
      }
      for (int i = 0; i < kNormSlots; ++i) {
        mbar_init(bar_nfull + 8 * i, 1);
        mbar_init(bar_nempty + 8 * i, 4 * qts);
      }
      mbar_init(bar_done, 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
      // an earlier block of the build gave up: do nothing.  FP32 filter: dense tiles take the tree
      if (BOUND) *status_p = (int)too_many(a, -1) | (int)too_many(a, 0) ? 2 : a.give_up ? 1 : 0;
      else *status_p = *reinterpret_cast<volatile int*>(a.err) != 0 ? 2 : 0;
    }
    __syncwarp();
  } else if (warp == 4 * QT + 1) {  // MMA warp: tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)Plan::kTotal));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const bool stopped = *status != 0;  // block-uniform: read after the barrier, not written before the next

  if (warp < 4 * QT) {
    // ------------------------------------------------ epilogue: a thread per row
    const int qt = warp >> 2, quarter = warp & 3;
    const uint32_t tlane = (uint32_t)(quarter * 32) << 16;
    const int row = q0 + qt * kBM + quarter * 32 + lane;  // row of the leaf
    const bool live = row < nq;
    const int64_t pos = lo + row;  // position in the tree's order
    const int qid = live ? a.perm[pos] : -1;
    const float myn = METRIC == KNN_METRIC_EUCLIDEAN && live ? a.np[pos] : 0.f;
    const float mydl = BOUND && live ? a.dp[pos] : 0.f;
    if (!stopped && qt < qts) {
      // the row's 16-bit elements into tensor memory, two per 32-bit column
      const uint16_t* src = a.Xp + (size_t)(live ? pos : lo) * a.ldr;
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          uint4 q = make_uint4(0u, 0u, 0u, 0u);
          const int e = ch * kKC + 8 * u;
          if (live && e < a.ldr) q = __ldg(reinterpret_cast<const uint4*>(src + e));
          v[4 * u] = q.x;
          v[4 * u + 1] = q.y;
          v[4 * u + 2] = q.z;
          v[4 * u + 3] = q.w;
        }
        tmem_st32(tmem + tlane + (uint32_t)(Plan::kA0 + qt * Plan::kA + ch * 32), v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();  // queries in place: MMAs may start
    if (!stopped && qt < qts) {
      const float kInf = __int_as_float(0x7F800000);
      const float kMaxF = __int_as_float(0x7F7FFFFF);
      unsigned char* mine = warp_area + (size_t)warp * kWarpBytes;
      unsigned char* dump = mine + lane * kDumpStride;                 // this row's slice
      uint32_t* bits = reinterpret_cast<uint32_t*>(mine + kWarpDump);  // [32][kBandWords]
      float* gm = reinterpret_cast<float*>(mine);                      // [32][kGS] during pass 0
      const size_t slot = (size_t)blockIdx.x * (kBM * QT) + warp * 32;  // the warp's rows in the scratch
      uint2* surv = a.surv + slot * kCap;
      uint2* mysurv = surv + lane * kCap;
      const int self = (int)(pos - blo);  // the row's own column (its leaf lies inside the block)
      int ca = 0, cb = nb;                // grouped leaves: the row's own leaf's columns
      if (a.glog) {
        int64_t s = lo, e = range.hi;
        for (int g = 0; g < (1 << a.glog); ++g) {
          const int64_t end = range.seg.off + node_lo(range.seg.n, range.seg.depth, range.j + g + 1);
          if (pos < end) {
            e = end;
            break;
          }
          s = end;
        }
        ca = (int)(s - blo);
        cb = (int)(e - blo);
      }
      // bound on the row's kq-th key (BOUND: scaled distance): its list tail, or the bounding pass's
      float tk = kInf;
      float cm_all = 0.f, dt_all = 0.f;  // largest |y|^2 and error bound met in the bounding pass
      bool over = false;                 // BOUND: the buffer was too small
      int cnt = 0;              // buffered survivors
      uint32_t have = FIRST ? 0u : 0xFFFFFFFFu;  // rows whose list holds something
      // later trees: the bitmap, for every row, of the columns in [band, band + kBand)
      // that hold an id of the row's list
      const int wrows = min(32, nq - (row - lane));  // rows of this warp (<= 0: none)
      auto set_band = [&](int band) {
        int32_t p[32];
        const int32_t* src = a.plist + (size_t)(pos - lane) * a.kq + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) p[i] = i < wrows && lane < a.kq ? __ldg(src + (size_t)i * a.kq) : -1;
        __syncwarp();
        for (int e = lane; e < 32 * kBandWords; e += 32) bits[e] = 0u;
        __syncwarp();
        const int32_t base = (int32_t)(blo + band);  // positions fit 31 bits
        const uint32_t width = (uint32_t)min(kBand, nb - band);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t c = (uint32_t)(p[i] - base);  // -1 and columns before the band wrap past width
          if (p[i] >= 0 && c < width) atomicOr(&bits[i * kBandWords + (c >> 5)], 1u << (c & 31));
        }
        __syncwarp();
      };
      const float scale = BOUND ? bound_scale(a) : 1.f;
      if (!FIRST) {
        if (BOUND) {
          if (live) tk = key_distance(a.rkey[(size_t)qid * a.kq + a.kq - 1], scale, a);
        } else {
          if (live) tk = from_orderable(a.akey[(size_t)qid * a.kq + a.kq - 1]);
        }
        if (!(tk < kInf)) tk = kInf;  // free slots
      }
      if (npre) {
#pragma unroll 8
        for (int e = 0; e < kGroups; ++e) gm[lane * kGS + e] = kInf;
      }
      bool ok = true;
#pragma unroll 1
      for (int s = 0; s < nsteps; ++s) {
        const bool pre = PRE && s < npre;
        const int t = s < npre ? s : s - npre;
        const int buf = s % NB;
        const uint32_t acc = (uint32_t)(qt * NB + buf);
        if (!FIRST && !pre && t * kTN % kBand == 0) set_band(t * kTN);
        if (METRIC == KNN_METRIC_EUCLIDEAN)
          ok = mbar_wait(bar_nfull + 8 * (s % kNormSlots), (uint32_t)(s / kNormSlots) & 1u, status, a.err);
        ok = ok && mbar_wait(bar_afull + 8 * acc, (uint32_t)(s / NB) & 1u, status, a.err);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const float* tn = tnorms + (s % kNormSlots) * (kTN + 4);
        const float cm = METRIC == KNN_METRIC_EUCLIDEAN ? tn[kTN] : 0.f;
        const float dt = BOUND ? tn[kTN + 1] : 0.f;
        float thr = kMaxF;  // the row's filter bound
        if (BOUND) {
          const float r = (tk + mydl + dt) * (1.f + a.g);
          thr = fminf((r * r + a.g1 * (myn + cm)) - myn, kMaxF);  // inf: every column
        } else if (tk < kInf) {
          if (METRIC == KNN_METRIC_EUCLIDEAN) thr = fminf((tk - myn) + kSlack * (fabsf(tk) + myn + cm), kMaxF);
          else thr = fminf((tk - 1.f) + kSlack * (fabsf(tk) + 2.f), kMaxF);
        }
        const uint64_t thr2 = pack2(__float_as_uint(thr), __float_as_uint(thr));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c0 = t * kTN + h * 32;  // the slice's first column
          uint32_t v[32];
          tmem_ld32(tmem + tlane + acc * kTN + (uint32_t)(h * 32), v);
          tmem_wait_ld(v);
          if (h == 1) {  // the accumulator is free
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_aempty + 8 * acc);
          }
          const ulonglong2* n4 = reinterpret_cast<const ulonglong2*>(tn + h * 32);  // four columns each
          // last use of the tile's norms by this warp (after the reads below)
          auto norms_done = [&]() {
            if (METRIC == KNN_METRIC_EUCLIDEAN && h == 1) {
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_nempty + 8 * (s % kNormSlots));
            }
          };
          const int own = self - c0;
          const int lim = nb - c0;  // columns of the block from c0 on
          if (pre) {
            // smallest key' of the slice, the row's own column and the columns
            // past the block left out, into the slice's group
            cm_all = fmaxf(cm_all, cm);
            dt_all = fmaxf(dt_all, dt);
            float big[4] = {-kInf, -kInf, -kInf, -kInf};  // of -key', per eight columns
            if (__any_sync(0xFFFFFFFFu, own >= 0 && own < 32) || lim < 32) {
#pragma unroll
              for (int c = 0; c < 32; ++c) v[c] = c == own || c >= lim ? 0xFF800000u : v[c];  // -inf: never the smallest
            }
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              uint32_t d[4] = {v[c], v[c + 1], v[c + 2], v[c + 3]};
              if (METRIC == KNN_METRIC_EUCLIDEAN) {
                const ulonglong2 n = n4[c >> 2];
                unpack2(fma2(pack2(0x40000000u, 0x40000000u), pack2(d[0], d[1]), n.x), d[0], d[1]);
                unpack2(fma2(pack2(0x40000000u, 0x40000000u), pack2(d[2], d[3]), n.y), d[2], d[3]);
              }
              float& b = big[c >> 3];
#pragma unroll
              for (int e = 0; e < 4; ++e) b = fmaxf(b, __uint_as_float(d[e]));
            }
            norms_done();
            float* group = gm + lane * kGS;
            const int slice = 2 * s + h;
            if (gw == 32) {
              float& x = group[slice & (kGroups - 1)];
              x = fminf(x, -fmaxf(fmaxf(big[0], big[1]), fmaxf(big[2], big[3])));
            } else if (gw == 16) {
              float* x = group + ((2 * slice) & (kGroups - 1));
              x[0] = fminf(x[0], -fmaxf(big[0], big[1]));
              x[1] = fminf(x[1], -fmaxf(big[2], big[3]));
            } else {
              float* x = group + ((4 * slice) & (kGroups - 1));
#pragma unroll
              for (int e = 0; e < 4; ++e) x[e] = fminf(x[e], -big[e]);
            }
            if (h == 1 && s == npre - 1) {
              // bound per row: the kq-th smallest of its group minima (kBoundRows
              // rows interleaved).  Each row's 64 minima: lanes' first halves sorted
              // ascending, second halves descending, their lane-wise minima are
              // the 32 smallest (a bitonic sequence), merged.
              __syncwarp();
              float bound = kInf;
#pragma unroll 1
              for (int i0 = 0; i0 < 32; i0 += kBoundRows) {
                float x[kBoundRows], y[kBoundRows];
#pragma unroll
                for (int i = 0; i < kBoundRows; ++i) {
                  x[i] = gm[(i0 + i) * kGS + lane];
                  y[i] = gm[(i0 + i) * kGS + 32 + lane];
                }
#pragma unroll 1
                for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll 1
                  for (int m = size >> 1; m >= 1; m >>= 1) {
                    const bool keep_min = ((lane & size) == 0) == ((lane & m) == 0);
#pragma unroll
                    for (int i = 0; i < kBoundRows; ++i) {
                      const float ox = __shfl_xor_sync(0xFFFFFFFFu, x[i], m);
                      const float oy = __shfl_xor_sync(0xFFFFFFFFu, y[i], m);
                      x[i] = keep_min ? fminf(x[i], ox) : fmaxf(x[i], ox);
                      y[i] = keep_min ? fmaxf(y[i], oy) : fminf(y[i], oy);
                    }
                  }
                }
#pragma unroll
                for (int i = 0; i < kBoundRows; ++i) x[i] = fminf(x[i], y[i]);
#pragma unroll 1
                for (int m = 16; m >= 1; m >>= 1) {
                  const bool keep_min = (lane & m) == 0;
#pragma unroll
                  for (int i = 0; i < kBoundRows; ++i) {
                    const float o = __shfl_xor_sync(0xFFFFFFFFu, x[i], m);
                    x[i] = keep_min ? fminf(x[i], o) : fmaxf(x[i], o);
                  }
                }
#pragma unroll
                for (int i = 0; i < kBoundRows; ++i) {
                  const float b = __shfl_sync(0xFFFFFFFFu, x[i], a.kq - 1);
                  if (lane == i0 + i) bound = b;
                }
              }
              // key' -> key units, widened past the rounding of both
              const float cap = BOUND ? minimum_distance(bound + myn + a.g1 * (myn + cm_all), mydl + dt_all, scale, a) :  METRIC == KNN_METRIC_EUCLIDEAN
                                    ? (bound + myn) + kSlack * (fabsf(bound) + 2.f * myn + cm_all)
                                    : (bound + 1.f) + kSlack * (fabsf(bound) + 2.f);
              if (cap < tk) tk = cap;
              __syncwarp();
            }
          } else {
            // bit c of neg = sign of thr - key'_c, shifted in from the highest column
            // down, in four independent chains of eight columns
            uint32_t part[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int c = 4; c >= 0; c -= 4)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int e = 8 * q + c;
                // -key' = 2 x.y - |y|^2 (EUCLIDEAN) or x.y (COSINE)
                uint64_t lo2 = pack2(v[e], v[e + 1]), hi2 = pack2(v[e + 2], v[e + 3]);
                if (METRIC == KNN_METRIC_EUCLIDEAN) {
                  const ulonglong2 n = n4[e >> 2];
                  lo2 = fma2(pack2(0x40000000u, 0x40000000u), lo2, n.x);
                  hi2 = fma2(pack2(0x40000000u, 0x40000000u), hi2, n.y);
                }
                uint32_t s0, s1, s2, s3;
                unpack2(add2(thr2, lo2), s0, s1);
                unpack2(add2(thr2, hi2), s2, s3);
                part[q] = __funnelshift_l(s3, part[q], 1);
                part[q] = __funnelshift_l(s2, part[q], 1);
                part[q] = __funnelshift_l(s1, part[q], 1);
                part[q] = __funnelshift_l(s0, part[q], 1);
              }
            const uint32_t neg = part[0] | (part[1] << 8) | (part[2] << 16) | (part[3] << 24);
            norms_done();
            uint32_t m = live ? ~neg : 0u;
            if (own >= 0 && own < 32) m &= ~(1u << own);
            if (lim < 32) m &= lim <= 0 ? 0u : (1u << lim) - 1u;
            if (a.glog) {  // grouped leaves: the row's own leaf's columns only
              const int lo_c = min(max(ca - c0, 0), 32), hi_c = min(max(cb - c0, 0), 32);
              m &= (uint32_t)(((1ull << hi_c) - 1ull) ^ ((1ull << lo_c) - 1ull));
        }
            if (!FIRST) m &= ~bits[lane * kBandWords + (c0 % kBand) / 32];
            const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, m);
            if (BOUND) {
              if (any) {
                over = over || cnt + __popc(m) > kCap;
                for (uint32_t left = over ? 0u : m; left; left &= left - 1) mysurv[cnt++].y = (uint32_t)(c0 + __ffs(left) - 1);
              }
            } else if (any) {
              // the products through shared memory (a lane cannot index its registers);
              // then every lane appends its own survivors
#pragma unroll
              for (int c = 0; c < 32; c += 4)
                *reinterpret_cast<uint4*>(dump + 4 * c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
              for (uint32_t left = m; left; left &= left - 1) {
                const int c = __ffs(left) - 1;
                mysurv[cnt++] = make_uint2(*reinterpret_cast<const uint32_t*>(dump + 4 * c), (uint32_t)(c0 + c));
              }
            }
          }
        }
        // a buffer too full for another tile is merged here (rare), with the
        // other well filled ones
        if (BOUND || pre || !__any_sync(0xFFFFFFFFu, cnt > kFlushAt)) continue;
        const uint32_t rows = __ballot_sync(0xFFFFFFFFu, cnt >= kFlushMin);
        tk = merge_survivors<METRIC>(a.akey, a.aid, a.np + blo, a.perm + blo, a.kq, surv, qid, myn, cnt, tk, have, rows);
        have |= rows;
        if ((rows >> lane) & 1u) cnt = 0;
      }
      if (BOUND) {
        const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, !ok ? 0u : over ? (uint32_t)nb : (uint32_t)cnt);
        if (lane == 0 && sum) atomicAdd(a.survivors, (unsigned long long)sum);
      }
      if (ok) a.count[slot + lane] = BOUND && over ? kOverflow : (uint32_t)cnt | (FIRST && ((have >> lane) & 1u) ? kListed : 0u);
    }
  } else {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();  // queries in place
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // Whole warps run these loops and one elected lane issues: the operands of
    // the TMA and MMA instructions stay in uniform registers.
    if (!stopped && warp == 4 * QT) {
      // ----------------------------------------------------------- producer
      const uint32_t ring0 = __shfl_sync(0xFFFFFFFFu, smem_u32(ring), 0);
      uint32_t q = 0;
      bool ok = true;
      // -|y|^2 of a tile's columns (EUCLIDEAN), -inf past the block, fetched a tile ahead
      const float kInf = __int_as_float(0x7F800000);
      float f0 = 0.f, f1 = 0.f, e0 = 0.f;
      auto fetch_norms = [&](int s) {
        const int c = (s < npre ? s : s - npre) * kTN + lane;
        f0 = c < nb ? a.np[blo + c] : kInf;
        f1 = c + 32 < nb ? a.np[blo + c + 32] : kInf;
        if (BOUND) e0 = fmaxf(c < nb ? a.dp[blo + c] : 0.f, c + 32 < nb ? a.dp[blo + c + 32] : 0.f);
      };
      if (METRIC == KNN_METRIC_EUCLIDEAN) fetch_norms(0);
      for (int s = 0; ok && s < nsteps; ++s) {
        const int t = s < npre ? s : s - npre;
        if (METRIC == KNN_METRIC_EUCLIDEAN) {
          const int slot = s % kNormSlots, round = s / kNormSlots;
          if (round > 0) ok = mbar_wait(bar_nempty + 8 * slot, (uint32_t)(round - 1) & 1u, status, a.err);
          if (!__all_sync(0xFFFFFFFFu, ok)) {
            ok = false;
            break;
          }
          float* tn = tnorms + slot * (kTN + 4);
          tn[lane] = -f0;
          tn[lane + 32] = -f1;
          if (BOUND) {
            const uint32_t worst = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(e0));
            if (lane == 0) tn[kTN + 1] = __uint_as_float(worst);
          }
          // norms are >= 0, so their bit patterns order as unsigned integers
          const float fm = fmaxf(f0 < kInf ? f0 : 0.f, f1 < kInf ? f1 : 0.f);
          const uint32_t big = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(fm));
          if (lane == 0) tn[kTN] = __uint_as_float(big);
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_nfull + 8 * slot);
          if (s + 1 < nsteps) fetch_norms(s + 1);
        }
        for (int ch = 0; ch < NCH; ++ch, ++q) {
          const uint32_t st = q % RING, round = q / RING;
          if (round > 0) ok = mbar_wait(bar_empty + 8 * st, (round - 1) & 1u, status, a.err);
          if (!__all_sync(0xFFFFFFFFu, ok)) {
            ok = false;
            break;
          }
          if (elect_one()) {
            mbar_expect_tx(bar_full + 8 * st, kBoxBytes);
            tma_load_box(ring0 + st * kBoxBytes, &bmap, ch * kKC, (int)(blo + (int64_t)t * kTN), bar_full + 8 * st);
          }
          __syncwarp();
        }
      }
      // the block's last loads land before it may end
      for (uint32_t d = q < (uint32_t)RING ? 0u : q - RING; d < q; ++d) {
        const uint64_t t0 = global_ns();
        while (!mbar_try_wait(bar_full + 8 * (d % RING), (d / RING) & 1u) && global_ns() - t0 < kWaitNs) {
        }
      }
    } else if (!stopped) {
      // ---------------------------------------------------------------- MMA
      const uint32_t ring0 = __shfl_sync(0xFFFFFFFFu, smem_u32(ring), 0);
      const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem, 0);
      uint32_t q = 0;
      bool ok = true;
      for (int s = 0; ok && s < nsteps; ++s) {
        // one query tile after the other: the next one's products need not wait for
        // this one's accumulator
        const int buf = s % NB, use = s / NB;
        for (int qt = 0; ok && qt < qts; ++qt) {
          if (use > 0) ok = mbar_wait(bar_aempty + 8 * (qt * NB + buf), (uint32_t)(use - 1) & 1u, status, a.err);
          const uint32_t d = tm + (uint32_t)((qt * NB + buf) * kTN);
          const uint32_t qa = tm + (uint32_t)(Plan::kA0 + qt * Plan::kA);
#pragma unroll
          for (int ch = 0; ch < NCH; ++ch) {
            const uint32_t st = (q + ch) % RING;
            if (qt == 0) ok = ok && mbar_wait(bar_full + 8 * st, ((q + ch) / RING) & 1u, status, a.err);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int steps = min(kKC / 16, a.ksteps - ch * (kKC / 16));
            const uint64_t b0 = desc_sw128(ring0 + st * kBoxBytes);
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < kKC / 16; ++kk)
                if (kk < steps)
                  umma_f16_ts(d, qa + ch * 32 + kk * 8, b0 + (uint64_t)(kk * 2), a.idesc, (ch | kk) != 0 ? 1u : 0u);
              if (qt == qts - 1) umma_commit(bar_empty + 8 * st);
              if (ch == NCH - 1) umma_commit(bar_afull + 8 * (qt * NB + buf));
            }
            __syncwarp();
          }
        }
        q += NCH;
      }
      // every issued product completes before tensor memory is freed
      if (elect_one()) umma_commit(bar_done);
      __syncwarp();
      const uint64_t t0 = global_ns();
      while (!mbar_try_wait(bar_done, 0) && global_ns() - t0 < kWaitNs) {
      }
    }
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  // FP32 filter: a block whose wait gave up leaves its tree to the dense tiles
  if (BOUND && tid == 0 && *status == 1) atomicMax(a.survivors, a.survivor_limit + 1ull);
  if (warp == 4 * QT + 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)Plan::kTotal));
  }
}

// The survivors that k_leaf_tc left, into the lists: a warp takes 32 rows (or an
// equal part of them, by gridDim.y), the rows with survivors (first tree: every
// row) kMergeRows at a time.  A kernel
// of its own, so that sorting and merging run at full occupancy instead of in
// the few warps that share an SM with the tiles, and never stall the products.
template <int METRIC, bool FIRST, int QT>
__global__ void __launch_bounds__(kBM * QT) k_leaf_tc_merge(const __grid_constant__ LeafTcArgs a) {
  const BlockRange range = block_range<QT>(a, a.block0 + blockIdx.x);
  const int lane = threadIdx.x & 31;
  const int row = range.q0 + (int)threadIdx.x;
  const bool live = row < (int)(range.hi - range.lo) && lane * (int)gridDim.y >> 5 == (int)blockIdx.y;
  if (*reinterpret_cast<volatile int*>(a.err) != 0) return;  // the build gave up: counts may be missing
  const size_t slot = (size_t)blockIdx.x * (kBM * QT) + threadIdx.x;
  uint32_t c = live ? a.count[slot] : 0u;
  const uint32_t rows = __ballot_sync(0xFFFFFFFFu, live && (FIRST ? c != kListed : c != 0u));
  if (rows == 0) return;
  const uint32_t have = FIRST ? __ballot_sync(0xFFFFFFFFu, (c & kListed) != 0u) : 0xFFFFFFFFu;
  const int64_t pos = range.lo + row;
  const int qid = live ? a.perm[pos] : -1;
  const float myn = METRIC == KNN_METRIC_EUCLIDEAN && live ? a.np[pos] : 0.f;
  merge_survivors<METRIC>(a.akey, a.aid, a.np + range.blo, a.perm + range.blo, a.kq, a.surv + (slot - lane) * kCap,
                          qid, myn, (int)(c & ~kListed), 0.f, have, rows);
}

// FP32 filter: the exact key (the reference's order) of every survivor, into
// the rows' lists.  A warp takes 32 rows (or an equal part of them, by gridDim.y)
// and packs their survivors, a lane each:
// the candidates' rows go through shared memory in slices (eight lanes read 128
// contiguous bytes; wider slices when there are fewer of them), the queries' come
// from L1.  Reading both straight from L1, a lane per survivor of one row, was
// bound by L1's one line per cycle: 300,000 x 128, 16 trees, leaf 512, 6.8 ms against
// 3.9.  A row whose buffer overflowed evaluates its whole block.
constexpr int kExactPitch = 128 + 16;            // row pitch of a 32-dim slice
constexpr int kExactBytes = 32 * kExactPitch;    // a warp's slice: 32 x 32, 16 x 64 or 8 x 128 dims
template <int METRIC, int QT>
__global__ void __launch_bounds__(kBM * QT, 10 / QT) k_leaf_tc_exact(const __grid_constant__ LeafTcArgs a,
                                                            float* __restrict__ rkey, uint32_t* __restrict__ rid) {
  __shared__ __align__(16) unsigned char slices[4 * QT * kExactBytes];
  const BlockRange range = block_range<QT>(a, a.block0 + blockIdx.x);
  const int lane = threadIdx.x & 31;
  unsigned char* slice = slices + (threadIdx.x >> 5) * kExactBytes;
  const int row = range.q0 + (int)threadIdx.x;
  const bool live = row < (int)(range.hi - range.lo) && lane * (int)gridDim.y >> 5 == (int)blockIdx.y;
  if (*reinterpret_cast<volatile int*>(a.err) != 0) return;  // a block gave up: dense tiles take the tree
  const float kInf = __int_as_float(0x7F800000);
  const size_t slot = (size_t)blockIdx.x * (kBM * QT) + threadIdx.x;
  const int64_t pos = range.lo + row;
  if (a.pair_counter) {  // statistics: pairs the filter decided on
    int64_t size = 0;
    if (live) {
      int64_t lo = range.lo, hi = range.hi;
      if (a.glog) {  // the row's own leaf
        for (int g = 0; g < (1 << a.glog); ++g) {
          hi = range.seg.off + node_lo(range.seg.n, range.seg.depth, range.j + g + 1);
          if (pos < hi) break;
          lo = hi;
        }
      }
      size = hi - lo - 1;
    }
    const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)size);
    if (lane == 0 && sum) atomicAdd(a.pair_counter, (unsigned long long)sum);
  }
  if (too_many(a, 0)) return;  // dense tiles follow (a later chunk's count may still decide so: they repeat this one)
  const uint32_t c = live ? a.count[slot] : 0u;
  if (!__any_sync(0xFFFFFFFFu, c != 0u)) return;
  const int qid = live ? a.perm[pos] : -1;
  uint2* surv = a.surv + (slot - lane) * kCap;

  // lane: the exact key of row r and the candidate at position p (valid lanes: the first m); cid: its id,
  // tail: the row's list tail
  auto keys = [&](int m, int r, int64_t p, int& cid, float& tail) {
    const bool valid = lane < m;
    const int id = __shfl_sync(0xFFFFFFFFu, qid, r);
    cid = valid ? __ldg(a.perm + p) : 0;
    tail = valid ? rkey[(size_t)id * a.k + a.k - 1] : -kInf;
    const float4* xq = reinterpret_cast<const float4*>(a.X + (size_t)(valid ? id : 0) * a.dpad);
    const int wlog = m <= 8 ? 7 : m <= 16 ? 6 : 5, width = 1 << wlog, pitch = 4 * width + 16;
    const int ulog = wlog - 2, c1 = lane & ((1 << ulog) - 1), r1 = lane >> ulog, rstep = 32 >> ulog;
    float total = 0.f, part = 0.f;
    for (int cd = 0; cd < a.d; cd += width) {
      const int dim = cd + 4 * c1;
      for (int i0 = 0; i0 < m; i0 += rstep) {
        const int i = i0 + r1;
        const int cand = __shfl_sync(0xFFFFFFFFu, cid, i & 31);
        if (i < m)
          cp_async16(smem_u32(slice + i * pitch + c1 * 16), a.X + (size_t)cand * a.dpad + (dim < a.dpad ? dim : 0),
                     dim < a.dpad ? 16 : 0);
      }
      asm volatile("cp.async.commit_group;\n" ::);
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncwarp();
      if (valid) {
        const float4* mine = reinterpret_cast<const float4*>(slice + lane * pitch);
        const int nu = (min(width, a.d - cd) + 3) / 4;
#pragma unroll 8
        for (int u = 0; u < nu; ++u) {
          const float4 w = mine[u];
          const float4 v = __ldg(xq + (cd >> 2) + u);
          part = acc_step<METRIC>(v.x, w.x, part);
          part = acc_step<METRIC>(v.y, w.y, part);
          part = acc_step<METRIC>(v.z, w.z, part);
          part = acc_step<METRIC>(v.w, w.w, part);
        }
        if (((cd + width) & 255) == 0 || cd + width >= a.d) {
          total = __fadd_rn(total, part);
          part = 0.f;
        }
      }
      __syncwarp();  // the slice is refilled next
    }
    float key = total;
    if (METRIC == KNN_METRIC_COSINE && valid) key = cosine_key(total, a.norms[id], a.norms[cid]);
    return key;
  };

  // the rows' survivors side by side: lane r holds the first slot of row r
  const int mine = c == kOverflow ? 0 : (int)c;
  int first = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xFFFFFFFFu, first, o);
    if (lane >= o) first += v;
  }
  const int all = __shfl_sync(0xFFFFFFFFu, first, 31);
  first -= mine;
  for (int e0 = 0; e0 < all; e0 += 32) {
    const int e = min(e0 + lane, all - 1);
    int r = 0;  // the last row whose first slot is at most e
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
      if (__shfl_sync(0xFFFFFFFFu, first, r + o) <= e) r += o;
    uint2* at = surv + (size_t)r * kCap + (e - __shfl_sync(0xFFFFFFFFu, first, r));
    int cid;
    float tail;
    const float key = keys(min(32, all - e0), r, range.blo + at->y, cid, tail);
    // the survivor's key and id take its place
    if (e0 + lane < all) *at = key <= tail ? make_uint2(orderable(key), (uint32_t)cid) : make_uint2(kNoKey, kNoId);
  }
  uint32_t rows = __ballot_sync(0xFFFFFFFFu, mine > 0);
  if (rows)
    merge_survivors<METRIC, true>(reinterpret_cast<uint32_t*>(rkey), rid, nullptr, nullptr, a.k, surv, qid, 0.f, mine,
                                  0.f, 0xFFFFFFFFu, rows);
  // overflowed rows: every column of the block
  for (rows = __ballot_sync(0xFFFFFFFFu, c == kOverflow); rows; rows &= rows - 1) {
    const int nb = (int)(range.bhi - range.blo), r = __ffs(rows) - 1;
    const int id = __shfl_sync(0xFFFFFFFFu, qid, r);
    WarpList<1> L;
    L.key[0] = lane < a.k ? rkey[(size_t)id * a.k + lane] : kInf;
    L.id[0] = lane < a.k ? rid[(size_t)id * a.k + lane] : kNoId;
    for (int e0 = 0; e0 < nb; e0 += 32) {
      int cid;
      float tk;
      uint32_t ti;
      const float key = keys(min(32, nb - e0), r, range.blo + min(e0 + lane, nb - 1), cid, tk);
      warp_list_get(L, a.k - 1, tk, ti);
      bool pass = e0 + lane < nb && cid != id && cand_less(key, (uint32_t)cid, tk, ti);
      if (!__any_sync(0xFFFFFFFFu, pass)) continue;
      const bool dup = warp_list_contains(L, (uint32_t)cid, a.k);
      pass = pass && !dup;
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, pass);
      if (bal) warp_list_insert_lanes(L, bal, key, (uint32_t)cid, kInf);
    }
    if (lane < a.k) {
      rkey[(size_t)id * a.k + lane] = L.key[0];
      rid[(size_t)id * a.k + lane] = L.id[0];
    }
    __syncwarp();
  }
}

// FP32 filter: a tree's 16-bit rows (see bound_scale): Xp = fp16(s (x - c)), np =
// |row|^2, dp bounds |s (x - c) - row| (L2).  A row that defeats the bound (a COSINE
// norm whose square leaves the FP32 range or is zero) becomes a zero row with dp =
// inf: always a survivor.  Infinite values and NaN, which have keys that no order
// ranks, leave the tree to the dense tiles.  Bound by the gather of the
// rows: a warp takes kCenterRows positions, whose leaves its lanes look up side by side.
constexpr int kCenterRows = 8;
__global__ void __launch_bounds__(256) k_center_operand(const __grid_constant__ LeafTcArgs a, uint16_t* __restrict__ Xp,
                                                        float* __restrict__ np, float* __restrict__ dp) {
  const int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kCenterRows;
  const int lane = threadIdx.x & 31;
  if (too_many(a, -1)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.survivors[0] = a.survivors[-1];
    return;
  }
  if (p0 >= a.n) return;
  const float scale = bound_scale(a);
  int32_t my_id = 0, my_cid = 0;
  float my_rx = 1.f, my_rc = 1.f;
  bool my_ok = true;
  if (lane < kCenterRows && p0 + lane < a.n) {
    const int64_t p = p0 + lane;
    const SegEntry e = a.segs.get(a.segs.of(p));
    const int64_t j = node_of(e.n, e.depth, p - e.off);
    const int64_t mid = e.off + (node_lo(e.n, e.depth, j) + node_lo(e.n, e.depth, j + 1)) / 2;
    my_id = __ldg(a.perm + p);
    my_cid = __ldg(a.perm + mid);
    if (a.metric == KNN_METRIC_COSINE) {
      const float nx = a.norms[my_id], nc = a.norms[my_cid];
      my_ok = nx > 8.67361738e-19f && nx < 1.15292150e18f;  // 2^-60, 2^60
      my_rx = __frcp_rn(nx);  // 0 or NaN: not finite
      my_rc = nc > 8.67361738e-19f && nc < 1.15292150e18f ? __frcp_rn(nc) : 0.f;
    }
  }
  const float base = a.metric == KNN_METRIC_COSINE ? scale * 4.76837158e-07f : 0.f;  // 2^-21: rounding of both unit rows
  const int rows = (int)min((int64_t)kCenterRows, a.n - p0);
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    const int32_t id = __shfl_sync(0xFFFFFFFFu, my_id, r), cid = __shfl_sync(0xFFFFFFFFu, my_cid, r);
    const float rx = __shfl_sync(0xFFFFFFFFu, my_rx, r), rc = __shfl_sync(0xFFFFFFFFu, my_rc, r);
    const float4* x4 = reinterpret_cast<const float4*>(a.X + (size_t)id * a.dpad);
    const float4* c4 = reinterpret_cast<const float4*>(a.X + (size_t)cid * a.dpad);
    uint16_t* out = Xp + (size_t)(p0 + r) * a.ldr;
    float err = 0.f, sq = 0.f;
    for (int i = 4 * lane; i < a.ldr; i += 128) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), c = x;  // rows are zero padded to dpad
      if (i < a.dpad) {
        x = __ldg(x4 + (i >> 2));
        c = __ldg(c4 + (i >> 2));
      }
      const float v[4] = {__fmul_rn(__fsub_rn(__fmul_rn(x.x, rx), __fmul_rn(c.x, rc)), scale),
                          __fmul_rn(__fsub_rn(__fmul_rn(x.y, rx), __fmul_rn(c.y, rc)), scale),
                          __fmul_rn(__fsub_rn(__fmul_rn(x.z, rx), __fmul_rn(c.z, rc)), scale),
                          __fmul_rn(__fsub_rn(__fmul_rn(x.w, rx), __fmul_rn(c.w, rc)), scale)};
      uint32_t h[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const __half y = __float2half_rn(v[q]);
        h[q] = __half_as_ushort(y);
        const float f = __half2float(y), t = __fsub_rn(v[q], f);
        err = __fmaf_rn(t, t, err);
        sq = __fmaf_rn(f, f, sq);
      }
      *reinterpret_cast<uint2*>(out + i) = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      err = __fadd_rn(err, __shfl_xor_sync(0xFFFFFFFFu, err, off));
      sq = __fadd_rn(sq, __shfl_xor_sync(0xFFFFFFFFu, sq, off));
    }
    // the subtraction's own rounding: 2^-23 of the row
    const float bound = __fsqrt_rn(err) * (1.f + 1.f / 1024.f) + __fsqrt_rn(sq) * 1.1920929e-07f + base;
    const bool usable = __shfl_sync(0xFFFFFFFFu, my_ok ? 1 : 0, r) != 0;
    const bool good = usable && bound < __int_as_float(0x7F800000) && sq < __int_as_float(0x7F800000);
    if (!good)
      for (int i = 4 * lane; i < a.ldr; i += 128) *reinterpret_cast<uint2*>(out + i) = make_uint2(0u, 0u);
    if (lane == 0) {
      if (!(rx > 0.f) || (usable && !good)) atomicMax(a.survivors, a.survivor_limit + 1ull);
      np[p0 + r] = good ? sq : 0.f;
      dp[p0 + r] = good ? bound : __int_as_float(0x7F800000);
    }
  }
}

// inv[order[i]] = i: the position of each point in a tree's order.
__global__ void k_inverse_order(const int32_t* __restrict__ order, int64_t n, int32_t* __restrict__ inv) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    inv[order[i]] = (int32_t)i;
}

__device__ __forceinline__ uint16_t to_operand(float v, bool f16) {
  return f16 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float from_operand(uint16_t b, bool f16) {
  return f16 ? __half2float(__ushort_as_half(b)) : __bfloat162float(__ushort_as_bfloat16(b));
}

// 16-bit operand copy: rows of ldr BF16 or FP16 values (zero padded), COSINE
// rows divided by their FP32 norm first; norms2 = |row|^2 of the rounded
// values (EUCLIDEAN).  FP16 EUCLIDEAN rows are first multiplied by the power
// of two 2^e that brings the largest |x| (maxabs) into [2^14, 2^15), inside
// the FP16 range: a power-of-two scale is exact, scales every key of the tile
// stage by the same 2^2e and so keeps its ranking (the re-rank uses X).  With perm,
// output row i is row perm[i].  A row with infinite values or NaN becomes a zero row with
// an infinite norm (COSINE: a key of 1): products with it would give keys of the form
// inf - inf, whose order is not defined, and it is no finite row's neighbour.
__global__ void k_to_operand(const float* __restrict__ X, int64_t n, int d, int dpad, int ldr, int metric, bool f16,
                             const unsigned int* __restrict__ maxabs, const float* __restrict__ norms,
                             const int32_t* __restrict__ perm, uint16_t* __restrict__ Xb, float* __restrict__ norms2) {
  const int64_t out = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (out >= n) return;
  const int64_t row = perm ? perm[out] : out;
  float scale = 1.f;
  if (metric == KNN_METRIC_COSINE) {
    const float nr = norms[row];
    scale = nr > 0.f ? __frcp_rn(nr) : 0.f;
  } else if (f16) {
    const float m = __uint_as_float(*maxabs);
    int e = 0;
    if (m > 0.f && m < __int_as_float(0x7F800000)) {
      frexpf(m, &e);  // m in [2^(e-1), 2^e)
      e = 15 - e;     // m * 2^(15-e) in [2^14, 2^15)
      e = max(-126, min(126, e));
    }
    scale = ldexpf(1.f, e);
  }
  float s = 0.f;
  bool finite = true;
  for (int c = lane; c < ldr; c += 32) {
    const float v = c < d ? X[(size_t)row * dpad + c] : 0.f;
    finite &= fabsf(v) < __int_as_float(0x7F800000);
    const uint16_t b = to_operand(__fmul_rn(v, scale), f16);
    Xb[(size_t)out * ldr + c] = b;
    const float f = from_operand(b, f16);
    s = __fmaf_rn(f, f, s);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, off));
  if (!__all_sync(0xFFFFFFFFu, finite)) {
    for (int c = lane; c < ldr; c += 32) Xb[(size_t)out * ldr + c] = 0;
    s = __int_as_float(0x7F800000);
  }
  if (lane == 0) norms2[out] = s;
}

// A tree's order: Xp[i] = Xb[perm[i]], np[i] = norms2[perm[i]]; one thread per
// 16-byte unit (units per row: ldr / 8).
__global__ void __launch_bounds__(256) k_permute_operand(const uint4* __restrict__ Xb,
                                                         const float* __restrict__ norms2,
                                                         const int32_t* __restrict__ perm, int64_t n, int units,
                                                         uint4* __restrict__ Xp, float* __restrict__ np) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n * units) return;
  const int64_t i = g / units;
  const int u = (int)(g - i * units);
  const int32_t id = __ldg(perm + i);
  Xp[g] = __ldg(Xb + (size_t)id * units + u);
  if (u == 0) np[i] = norms2[id];
}

// Positions in a tree's order of every entry of every point's list, rows in
// that order too (-1: empty): plist[p][e] = inv[aid[perm[p]][e]].
__global__ void __launch_bounds__(256) k_list_positions(const uint32_t* __restrict__ aid,
                                                        const int32_t* __restrict__ perm,
                                                        const int32_t* __restrict__ inv, int64_t n, int kq,
                                                        int32_t* __restrict__ plist) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n * kq) return;
  const int64_t p = g / kq;
  const uint32_t id = aid[(size_t)__ldg(perm + p) * kq + (int)(g - p * kq)];
  plist[g] = id < (uint64_t)n ? __ldg(inv + id) : -1;
}

// Exact FP32 keys (the reference's order) of each point's kq approximate
// candidates; the best k become the list, all flagged new.  One warp per point:
// the candidate rows are staged 64 dims at a time by 16-byte cp.async into an
// xor-swizzled tile (lane r reads row r conflict-free), one lane per candidate.
template <int METRIC>
__global__ void __launch_bounds__(256) k_rerank(const float* __restrict__ X, int64_t n, int d, int dpad,
                                                int k, int kq, const float* __restrict__ norms,
                                                const uint32_t* __restrict__ aid,
                                                float* __restrict__ rkey, uint32_t* __restrict__ rid) {
  extern __shared__ __align__(16) float rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  float* xq = rsm + (size_t)warp * (dpad + 32 * 64 + 32);
  float* rows = xq + dpad;
  uint32_t* ids = reinterpret_cast<uint32_t*>(rows + 32 * 64);
  if (i >= n) return;
  const float kInf = __int_as_float(0x7F800000);
  const float4* xr = reinterpret_cast<const float4*>(X + (size_t)i * dpad);
  for (int c = lane; c < (dpad >> 2); c += 32) reinterpret_cast<float4*>(xq)[c] = xr[c];
  // an id outside [0, n) is an empty entry
  uint32_t cj = lane < kq ? aid[(size_t)i * kq + lane] : kNoId;
  if (cj >= (uint64_t)n) cj = kNoId;
  const bool valid = cj != kNoId;
  ids[lane] = cj;
  __syncwarp();
  float total = 0.f, part = 0.f;
  const int half = lane >> 4, c4 = lane & 15;
  for (int cd = 0; cd < d; cd += 64) {
    const int dim = cd + 4 * c4;
    for (int r = half; r < 32; r += 2) {
      const uint32_t id = ids[r];
      const bool ok = id != kNoId && dim < dpad;
      const float* src = X + (size_t)(id != kNoId ? id : 0) * dpad + (dim < dpad ? dim : 0);
      cp_async16(smem_u32(rows + r * 64 + ((c4 ^ (r & 7)) << 2)), src, ok ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp();
    const int lim = min(64, d - cd);
    const float* myrow = rows + lane * 64;
    for (int q4 = 0; q4 < (lim + 3) >> 2; ++q4) {
      const float4 cv = *reinterpret_cast<const float4*>(myrow + ((q4 ^ (lane & 7)) << 2));
      const float4 qv = *reinterpret_cast<const float4*>(xq + cd + 4 * q4);
      part = acc_step<METRIC>(qv.x, cv.x, part);
      part = acc_step<METRIC>(qv.y, cv.y, part);
      part = acc_step<METRIC>(qv.z, cv.z, part);
      part = acc_step<METRIC>(qv.w, cv.w, part);
    }
    if (((cd + 64) & 255) == 0 || cd + 64 >= d) {
      total = __fadd_rn(total, part);
      part = 0.f;
    }
    __syncwarp();
  }
  float key = total;
  if (METRIC == KNN_METRIC_COSINE) key = valid ? cosine_key(total, norms[i], norms[cj]) : kInf;
  if (!valid) key = kInf;
  float kk = key;
  uint32_t ii = valid ? cj : kNoId;
  warp_bitonic_sort32(kk, ii);
  if (lane < k) {
    rkey[(size_t)i * k + lane] = kk;
    rid[(size_t)i * k + lane] = ii;
  }
}

namespace {

template <int NCH, int QT>
size_t leaf_tc_smem() {
  return 1024 + (size_t)kRing * kBoxBytes + (size_t)4 * QT * kWarpBytes + kNormBytes +
         8 * (2 * kRing + 2 * QT * TmemPlan<NCH, QT>::kNB + 2 * kNormSlots + 1) + 16;
}

// 2-D map of the 16-bit rows [n][ldr]: boxes of 64 rows x 64 elements, zeros
// outside (past the last row and past column ldr).
bool operand_map(const void* Xp, int64_t n, int ldr, bool f16, CUtensorMap* map) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Encode>(f);
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)ldr, (cuuint64_t)n};
  const cuuint64_t strides[1] = {(cuuint64_t)ldr * 2};
  const cuuint32_t box[2] = {kKC, kTN};
  const cuuint32_t one[2] = {1, 1};
  return encode(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                const_cast<void*>(Xp), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A tree's tiles, `rows` rows at a time, each chunk followed by its merge
// (BOUND: into the exact lists rkey / rid).
template <int METRIC, bool BOUND, bool FIRST, bool PRE, int NCH, int QT>
void launch_tc(const CUtensorMap& map, LeafTcArgs t, int64_t blocks, int64_t rows, float* rkey, uint32_t* rid,
               cudaStream_t st, LaunchLog& log) {
  const size_t smem = leaf_tc_smem<NCH, QT>();
  cudaFuncSetAttribute(k_leaf_tc<METRIC, BOUND, FIRST, PRE, NCH, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem);
  const int64_t chunk = rows / (kBM * QT);
  for (t.block0 = 0; t.block0 < blocks; t.block0 += chunk) {
    const unsigned grid = (unsigned)std::min(chunk, blocks - t.block0);
    k_leaf_tc<METRIC, BOUND, FIRST, PRE, NCH, QT><<<grid, 64 + 128 * QT, smem, st>>>(map, t);
    // Few rows leave most of the chip idle in the kernels after the tiles, where a
    // warp works through its 32 rows' survivors at the latency of its loads: each
    // warp's rows are spread over up to eight warps until 8,000 are there (a chip
    // holds 5,920; FP32, 36,155 x 246, 11 trees, leaf 104: one warp 4.09 ms, two 3.07,
    // four 2.68, eight 2.56; 300,000 x 128, 16 trees, leaf 512: 10.78, 10.81, 11.30,
    // 12.38; BF16 products, 5,206 x 23, 5 trees, leaf 77: 0.45, 0.39, 0.37, 0.35).
    dim3 split(grid, 1);
    while (split.y < 8 && 4 * QT * grid * split.y < 8000) split.y *= 2;
    if (!BOUND) k_leaf_tc_merge<METRIC, FIRST, QT><<<split, kBM * QT, 0, st>>>(t);
    else if (t.metric == KNN_METRIC_COSINE) k_leaf_tc_exact<KNN_METRIC_COSINE, QT><<<split, kBM * QT, 0, st>>>(t, rkey, rid);
    else k_leaf_tc_exact<KNN_METRIC_EUCLIDEAN, QT><<<split, kBM * QT, 0, st>>>(t, rkey, rid);
    log.add(2);
  }
}
template <int METRIC, bool BOUND, bool FIRST, bool PRE>
void launch_tc_tiles(int qt, int nch, const CUtensorMap& map, const LeafTcArgs& t, int64_t blocks, int64_t rows,
                     float* rkey, uint32_t* rid, cudaStream_t st, LaunchLog& log) {
  if (qt == 2 && nch == 1) launch_tc<METRIC, BOUND, FIRST, PRE, 1, 2>(map, t, blocks, rows, rkey, rid, st, log);
  else if (qt == 2) launch_tc<METRIC, BOUND, FIRST, PRE, 2, 2>(map, t, blocks, rows, rkey, rid, st, log);
  else if (nch == 1) launch_tc<METRIC, BOUND, FIRST, PRE, 1, 1>(map, t, blocks, rows, rkey, rid, st, log);
  else if (nch == 2) launch_tc<METRIC, BOUND, FIRST, PRE, 2, 1>(map, t, blocks, rows, rkey, rid, st, log);
  else if (nch == 3) launch_tc<METRIC, BOUND, FIRST, PRE, 3, 1>(map, t, blocks, rows, rkey, rid, st, log);
  else launch_tc<METRIC, BOUND, FIRST, PRE, 4, 1>(map, t, blocks, rows, rkey, rid, st, log);
}
template <int METRIC, bool BOUND>
void launch_tc_tree(bool first, bool pre, int qt, int nch, const CUtensorMap& map, const LeafTcArgs& t, int64_t blocks,
                    int64_t rows, float* rkey, uint32_t* rid, cudaStream_t st, LaunchLog& log) {
  if (first) launch_tc_tiles<METRIC, BOUND, true, true>(qt, nch, map, t, blocks, rows, rkey, rid, st, log);
  else if (pre) launch_tc_tiles<METRIC, BOUND, false, true>(qt, nch, map, t, blocks, rows, rkey, rid, st, log);
  else launch_tc_tiles<METRIC, BOUND, false, false>(qt, nch, map, t, blocks, rows, rkey, rid, st, log);
}

}  // namespace

namespace {
// Query tiles per block and blocks per leaf (or per group of sibling leaves).
// Two query tiles share every candidate box, which halves the L2 reads (integer
// mixture, 8 trees, leaf 2048, tiles without the second bounding pass: 14.9 ms
// against 15.1 with one; 10M x 96 COSINE 194 against 199); one where leaves (or
// groups of them) fill a single tile, and above 128 dims, where two query tiles
// would take all of tensor memory.
struct TcShape {
  int qt, qtiles, glog;
};
TcShape tc_shape(int d, int64_t maxleaf, int tc_group) {
  TcShape s;
  s.glog = tc_group >= 4 ? 2 : tc_group == 2 ? 1 : 0;
  s.qt = d > 2 * kKC || s.glog || maxleaf <= kBM ? 1 : 2;
  s.qtiles = s.glog ? 1 : (int)((maxleaf + kBM * s.qt - 1) / (kBM * s.qt));
  return s;
}
}  // namespace

size_t umma_scratch_rows(const UmmaLeafArgs& a) {
  const TcShape s = tc_shape(a.d, a.maxleaf, a.tc_group);
  int64_t leaves = a.leaves >> s.glog;
  for (int t = 0; a.ftable && t < a.trees; ++t) leaves = std::max(leaves, a.fcount[t]);
  return (size_t)std::min<int64_t>(kChunkRows, leaves * s.qtiles * (kBM * s.qt));
}
int umma_block_rows(const UmmaLeafArgs& a) { return kBM * tc_shape(a.d, a.maxleaf, a.tc_group).qt; }
size_t umma_row_scratch_bytes() { return kCap * sizeof(uint2); }

int leaf_stage_umma(const UmmaLeafArgs& a, LaunchLog& log) {
  const int nch = (a.d + kKC - 1) / kKC;
  if (nch > 4 || a.kq > 32 || a.kq < a.k) return KNN_ERR_UNSUPPORTED;
  cudaStream_t st = a.stream;
  uint16_t* Xb = static_cast<uint16_t*>(a.Xb);
  // operand copy (FP16 EUCLIDEAN: the largest |x| first, for the row scale)
  if (a.f16 && a.metric == KNN_METRIC_EUCLIDEAN) {
    launch_max_abs(a.X, a.n, a.dpad, a.maxabs, st);
    log.add();
  }
  const int ldr = umma_row_stride(a.d);
  auto convert = [&](const int32_t* perm, uint16_t* rows, float* norms2) {
    k_to_operand<<<(unsigned)((a.n * 32 + 255) / 256), 256, 0, st>>>(a.X, a.n, a.d, a.dpad, ldr, a.metric, a.f16,
                                                                      a.maxabs, a.norms, perm, rows, norms2);
    log.add();
  };
  if (Xb) convert(nullptr, Xb, a.norms2);
  CUtensorMap map;
  if (!operand_map(a.Xp, a.n, ldr, a.f16, &map)) return KNN_ERR_CUDA;
  const int64_t leaves = a.leaves;
  // 2^glog sibling leaves per tile (the caller checks it is allowed)
  const TcShape shape = tc_shape(a.d, a.maxleaf, a.tc_group);
  const int qt = shape.qt, glog = shape.glog;
  if (glog && (a.ftable || (a.maxleaf << glog) > kBM)) return KNN_ERR_UNSUPPORTED;
  LeafTcArgs t{};
  t.Xp = static_cast<const uint16_t*>(a.Xp);
  t.np = a.np;
  t.segs = a.segs;
  t.akey = a.akey;
  t.aid = a.aid;
  t.err = a.err;
  t.surv = static_cast<uint2*>(a.surv);
  t.count = a.surv_count;
  t.n = a.n;
  t.idesc = idesc_for(a.f16);
  t.ldr = ldr;
  t.ksteps = (a.d + 15) / 16;
  t.k = a.k;
  t.kq = a.kq;
  t.qtiles = shape.qtiles;
  t.glog = glog;
  const int units = ldr / 8;
  for (int tr = 0; tr < a.trees; ++tr) {
    t.perm = a.perm + (size_t)tr * a.n;
    t.ftab = a.ftable ? a.ftable + 4 * a.foff[tr] : nullptr;
    const int64_t tleaves = a.ftable ? a.fcount[tr] : (leaves >> glog);
    if (tleaves <= 0) {
      if (a.kev) {
        cudaEventRecord(a.kev[2 * tr], st);
        cudaEventRecord(a.kev[2 * tr + 1], st);
      }
      continue;
    }
    const int64_t blocks = tleaves * t.qtiles;
    if (Xb) {
      k_permute_operand<<<(unsigned)((a.n * units + 255) / 256), 256, 0, st>>>(
          reinterpret_cast<const uint4*>(Xb), a.norms2, t.perm, a.n, units, static_cast<uint4*>(a.Xp), a.np);
      log.add();
    } else {
      convert(t.perm, static_cast<uint16_t*>(a.Xp), a.np);
    }
    if (tr > 0) {
      const int32_t* inv = a.tree_inv ? a.tree_inv + (size_t)tr * a.n : a.inv;
      if (!a.tree_inv) {
        k_inverse_order<<<(unsigned)std::min<int64_t>((a.n + 255) / 256, 148 * 16), 256, 0, st>>>(t.perm, a.n, a.inv);
        log.add();
      }
      k_list_positions<<<(unsigned)((a.n * a.kq + 255) / 256), 256, 0, st>>>(a.aid, t.perm, inv, a.n, a.kq, a.plist);
      log.add();
      t.plist = a.plist;
    }
    if (a.kev) cudaEventRecord(a.kev[2 * tr], st);
    const bool pre = tr < kPrepassTrees && a.maxleaf >= kPrepassMin;
    if (a.metric == KNN_METRIC_EUCLIDEAN)
      launch_tc_tree<KNN_METRIC_EUCLIDEAN, false>(tr == 0, pre, qt, nch, map, t, blocks, a.rows, nullptr, nullptr, st, log);
    else
      launch_tc_tree<KNN_METRIC_COSINE, false>(tr == 0, pre, qt, nch, map, t, blocks, a.rows, nullptr, nullptr, st, log);
    if (a.kev) cudaEventRecord(a.kev[2 * tr + 1], st);
  }
  // shared memory of k_rerank's eight warps; the attribute is the process's, so one value for all dims
  auto rerank_smem = [](int dpad) { return (size_t)8 * (dpad + 32 * 64 + 32) * sizeof(float); };
  const size_t rsm = rerank_smem(a.dpad);
  const int rsm_max = (int)rerank_smem(4 * kKC);
  const unsigned rgrid = (unsigned)((a.n + 7) / 8);
  if (a.metric == KNN_METRIC_EUCLIDEAN) {
    cudaFuncSetAttribute(k_rerank<KNN_METRIC_EUCLIDEAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, rsm_max);
    k_rerank<KNN_METRIC_EUCLIDEAN><<<rgrid, 256, rsm, st>>>(a.X, a.n, a.d, a.dpad, a.k, a.kq, a.norms, a.aid, a.rkey, a.rid);
  } else {
    cudaFuncSetAttribute(k_rerank<KNN_METRIC_COSINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, rsm_max);
    k_rerank<KNN_METRIC_COSINE><<<rgrid, 256, rsm, st>>>(a.X, a.n, a.d, a.dpad, a.k, a.kq, a.norms, a.aid, a.rkey, a.rid);
  }
  log.add();
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

// ---------------------------------------------------------- FP32 leaf filter --
size_t filter_scratch_rows(const FilterLeafArgs& a) {
  const TcShape s = tc_shape(a.d, a.maxleaf, a.tc_group);
  return (size_t)std::min<int64_t>(kChunkRows, (a.leaves >> s.glog) * s.qtiles * (kBM * s.qt));
}

// Group widths of 8, 16 and 32 start at 256, 513 and 1,025 columns, so groups times
// width reach 1.25 k at every size from minleaf on if they do at 256.
bool umma_bounds_first_tree(int64_t minleaf, int k) { return minleaf >= kPrepassMin && 8 * (k + k / 4) <= kPrepassMin; }

// Data that the 16-bit rows cannot tell apart (several scales within one leaf)
// would send most pairs down the survivors' path, at several times a dense
// tile's cost (400,000 x 256, leaf 1,000, all pairs: 415 ms against 64), so from
// an eighth of the pairs and 16 + k a row the dense tiles take over.
unsigned long long filter_survivor_limit(const FilterLeafArgs& a) {
  return (unsigned long long)a.n * (unsigned long long)(16 + a.k + a.maxleaf / 8);
}

bool filter_map(FilterLeafArgs* a) {
  CUtensorMap map;
  if (!operand_map(a->Xp, a->n, umma_row_stride(a->d), true, &map)) return false;
  static_assert(sizeof(map) == sizeof(a->map), "tensor map");
  memcpy(a->map, &map, sizeof(map));
  return true;
}

int leaf_stage_filtered(const FilterLeafArgs& a, LaunchLog& log) {
  const int nch = (a.d + kKC - 1) / kKC;
  if (nch > 4 || a.k > 32 || a.metric == KNN_METRIC_TAXICAB) return KNN_ERR_UNSUPPORTED;
  cudaStream_t st = a.stream;
  const TcShape shape = tc_shape(a.d, a.maxleaf, a.tc_group);
  const int ldr = umma_row_stride(a.d);
  if (a.metric == KNN_METRIC_EUCLIDEAN) {
    launch_max_abs(a.X, a.n, a.dpad, a.maxabs, st);
    log.add();
  }
  CUtensorMap map;
  memcpy(&map, a.map, sizeof(map));
  LeafTcArgs t{};
  t.Xp = static_cast<const uint16_t*>(a.Xp);
  t.np = a.np;
  t.dp = a.dp;
  t.segs = a.segs;
  t.aid = a.rid;
  t.err = reinterpret_cast<int*>(a.survivors + a.trees + 1 + kFilterErrGap);
  t.n = a.n;
  t.idesc = idesc_for(true);
  t.ldr = ldr;
  t.ksteps = (a.d + 15) / 16;
  t.k = t.kq = a.k;
  t.qtiles = shape.qtiles;
  t.glog = shape.glog;
  t.surv = static_cast<uint2*>(a.surv);
  t.count = a.count;
  t.X = a.X;
  t.norms = a.norms;
  t.rkey = a.rkey;
  t.maxabs = a.maxabs;
  t.pair_counter = a.pair_counter;
  t.give_up = a.give_up;
  t.g = (float)(2 * a.d + 64) * 5.9604644775390625e-08f;   // 2^-24
  t.g1 = (float)(a.d + 64) * 4.76837158203125e-07f;        // 2^-21: the tensor cores' sums are not rounded to nearest
  t.d = a.d;
  t.dpad = a.dpad;
  t.metric = a.metric;
  const int64_t blocks = (a.leaves >> shape.glog) * shape.qtiles;
  cudaMemsetAsync(a.survivors, 0, sizeof(unsigned long long) * filter_counters(a.trees), st);
  t.survivor_limit = filter_survivor_limit(a);
  for (int tr = a.first_tree; tr < a.trees; ++tr) {
    if (a.kev) cudaEventRecord(a.kev[2 * tr], st);
    t.perm = a.perm + (size_t)tr * a.n;
    t.survivors = a.survivors + tr + 1;
    k_center_operand<<<(unsigned)((a.n + 8 * kCenterRows - 1) / (8 * kCenterRows)), 256, 0, st>>>(t, static_cast<uint16_t*>(a.Xp), a.np, a.dp);
    log.add();
    if (tr > 0) {
      k_list_positions<<<(unsigned)((a.n * a.k + 255) / 256), 256, 0, st>>>(a.rid, t.perm, a.tree_inv + (size_t)tr * a.n,
                                                                            a.n, a.k, a.plist);
      log.add();
      t.plist = a.plist;
    }
    const bool pre = tr < kPrepassTrees && a.maxleaf >= kPrepassMin;
    launch_tc_tree<KNN_METRIC_EUCLIDEAN, true>(tr == 0, pre, shape.qt, nch, map, t, blocks, a.rows, a.rkey, a.rid, st, log);
    const int rc = a.dense_tree(tr, t.survivors, t.survivor_limit);
    if (rc) return rc;
    if (a.kev) cudaEventRecord(a.kev[2 * tr + 1], st);
  }
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

}  // namespace knn
