// Neighbour propagation, one Jacobi step: N'(i) = k best of N(i) u N(N(i)) \ {i}.
//
// Replaces propagate{Euclidean,Taxicab,Cosine}Kernel and the host loop
// (euclideandistancematrixgpu.cu:1033-1935, :1937-1977).  The reference marks
// N(N(i)) in an N-byte bitmap per point, clears N(i) and i, scans the bitmap and
// histogram-selects; here one warp owns one point:
//   * the k x k neighbour-of-neighbour ids are read all at once (four loads in
//     flight per lane), deduplicated in a per-warp shared-memory hash set
//     seeded with i and N(i), and compacted into a candidate array;
//   * the candidates' rows are staged by cp.async in 256-byte row slices (32
//     rows per stage, padded pitch so the per-lane row reads are conflict-free
//     at compile-time offsets); FP16 inputs are gathered as FP16 (the
//     conversion to FP32 is exact, so the keys are unchanged);
//   * each lane computes one key in the reference's order and the batch's
//     survivors are merged into the warp-held sorted list (bitonic via shuffles).
// Up to 1024 dims k_propagate_filtered, below, first rejects the candidates that
// cannot enter from 16-bit rows with rigorous bounds, and computes exact keys only
// for the rest: the same result.  k_propagate, every key exact, remains for longer
// rows, lists too long for the filter's shared memory, shapes where it is the faster one
// (prop_filter_pays), and ranges so small that preparing all points' 16-bit rows
// would cost more than the range.
// "New" flags: a pair (a, j) is skipped when a was already in N(i) and j already
// in N(a) before the previous step.  Such a j was a candidate of i in that step
// and lost to k better entries (or is listed), and N(i) only improves, so it
// cannot enter now: the result is identical to evaluating every pair.  The
// candidate set does not depend on the order of discovery, and the list keeps
// the k best of the set by (key, id), so the result does not either.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "knn_internal.cuh"
#include "knn_kernels.cuh"

namespace knn {

namespace {
constexpr int kPropMaxWarps = 8;
constexpr size_t kPropSmemBudget = 200 * 1024;
constexpr int kSliceBytes = 256;  // bytes of one candidate row per stage (16 x 16 B)
constexpr int kRowStride = kSliceBytes + 16;  // padded row pitch of the staging buffer
constexpr int kGatherUnroll = 4;  // neighbour-list entries in flight per lane
constexpr int kFiltPitch = 128 + 16;  // row pitch of the filtered step's exact slices (32 rows of 32 dims)
constexpr int kFiltMaxDim = 1024;     // a query's 16-bit row fits the warp's registers

__device__ __forceinline__ bool hash_insert(int32_t* H, int hbits, int32_t id) {
  const uint32_t size = 1u << hbits;
  uint32_t slot = ((uint32_t)id * 2654435761u) >> (32 - hbits);
  for (uint32_t probe = 0; probe < size; ++probe) {
    const int32_t prev = atomicCAS(&H[slot], -1, id);
    if (prev == -1) return true;
    if (prev == id) return false;
    slot = (slot + 1) & (size - 1);
  }
  return false;  // unreachable: the table holds twice the most insertions
}

inline int round_up(int v, int m) { return (v + m - 1) / m * m; }

}  // namespace

int prop_hash_bits(int k) {
  const int need = 2 * (k * k + k + 1);
  int b = 5;
  while ((1 << b) < need) ++b;
  return b;
}

// hash set (with two buffers: also the second row-slice buffer, since the
// hash is done with before the first row is staged) | candidates [k*k] | N(i)
// ids and flags | query row (float, d rounded to 8) | the row-slice buffer
// (32 rows, padded pitch)
size_t prop_region0_bytes(int k, int nbuf) {
  const size_t h = (size_t)4 << prop_hash_bits(k);
  return nbuf == 2 ? std::max(h, (size_t)32 * kRowStride) : h;
}
size_t prop_warp_bytes(int k, int d, int nbuf) {
  size_t b = prop_region0_bytes(k, nbuf) + (size_t)4 * round_up(k * k, 32) + (size_t)8 * round_up(k, 32) +
             (size_t)4 * round_up(d, 8) + (size_t)32 * kRowStride;
  return (b + 15) & ~(size_t)15;
}

// HALF: rows are FP16 [n][ldr] (ldr % 8 == 0), else float32 [n][ldr] (ldr % 4 == 0);
// zero padded beyond d.  NBUF 2: the next stage's row slices load while the
// current stage is summed (used where the second buffer costs no warps per SM).
template <int METRIC, int KPL, bool HALF, int NBUF>
__global__ void __launch_bounds__(kPropMaxWarps * 32) k_propagate(
    const void* __restrict__ Xrows, int ldr, int64_t n, int64_t r0, int64_t cnt, int d, int k, int kw, int hbits,
    size_t warp_bytes, size_t region0, const float* __restrict__ norms, const int32_t* __restrict__ order,
    const float* __restrict__ key_in, const uint32_t* __restrict__ id_in,
    const uint32_t* __restrict__ flags_in, float* __restrict__ key_out,
    uint32_t* __restrict__ id_out, uint32_t* __restrict__ flags_out,
    unsigned long long* __restrict__ cand_counter) {
  using Elem = typename std::conditional<HALF, __half, float>::type;
  constexpr int kEPU = 16 / sizeof(Elem);            // elements per 16-byte unit
  constexpr int kCH = kSliceBytes / sizeof(Elem);    // dims per row slice (divides 256)
  extern __shared__ __align__(16) unsigned char smem[];
  const Elem* X = static_cast<const Elem*>(Xrows);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* base = smem + (size_t)warp * warp_bytes;
  const int hsize = 1 << hbits;
  const int kk = k * k;
  const int kr = (k + 31) & ~31;
  const int dq = (d + 7) & ~7;
  int32_t* H = reinterpret_cast<int32_t*>(base);
  uint32_t* Q = reinterpret_cast<uint32_t*>(base + region0);
  uint32_t* nbid = Q + ((kk + 31) & ~31);
  uint32_t* nbfl = nbid + kr;
  float* xq = reinterpret_cast<float*>(nbfl + kr);
  unsigned char* rows1 = reinterpret_cast<unsigned char*>(xq + dq);  // [32][kRowStride]
  unsigned char* rows0 = NBUF == 2 ? base : rows1;                    // over the hash set
  const float kInf = __int_as_float(0x7F800000);
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int nch = (d + kCH - 1) / kCH;
  unsigned long long evaluated = 0;

  const int wpb = blockDim.x >> 5;
  const int64_t nwarps = (int64_t)gridDim.x * wpb;
  // points (or order positions) r0 .. r0 + cnt - 1
  for (int64_t w = (int64_t)blockIdx.x * wpb + warp; w < cnt; w += nwarps) {
    const int32_t i = order ? order[r0 + w] : (int32_t)(r0 + w);
    WarpList<KPL> L;
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      uint32_t nid = kNoId, nfl = 0;
      if (e < k) {
        L.key[r] = key_in[(size_t)i * k + e];
        // an id outside [0, n) is an empty entry: kept out of the list and
        // never followed
        const uint32_t u = id_in[(size_t)i * k + e] & kIdMask;
        const bool ok = u < (uint64_t)n;
        L.key[r] = ok ? L.key[r] : kInf;
        L.id[r] = ok ? u : kNoId;
        nid = ok ? u : kNoId;
        nfl = flags_in ? ((flags_in[(size_t)i * kw + r] >> lane) & 1u) : 1u;
      } else {
        L.key[r] = kInf;
        L.id[r] = kNoId;
      }
      if (e < kr) {
        nbid[e] = nid;
        nbfl[e] = nfl;
      }
    }
    for (int s = lane; s < hsize; s += 32) H[s] = -1;
    {
      const Elem* xr = X + (size_t)i * ldr;
      for (int c = lane; c < dq; c += 32) xq[c] = c < d ? (float)xr[c] : 0.f;
    }
    __syncwarp();
    if (lane == 0) hash_insert(H, hbits, i);
#pragma unroll
    for (int r = 0; r < KPL; ++r)
      if (r * 32 + lane < k && L.id[r] != kNoId) hash_insert(H, hbits, (int32_t)L.id[r]);
    __syncwarp();
    const float ni = (METRIC == KNN_METRIC_COSINE) ? norms[i] : 0.f;

    // candidates: entry (s, t) of the flattened k x k neighbour lists, lane-strided
    int qn = 0;
    for (int e0 = 0; e0 < kk; e0 += 32 * kGatherUnroll) {
      uint32_t jj[kGatherUnroll];
      bool ok[kGatherUnroll];
#pragma unroll
      for (int u = 0; u < kGatherUnroll; ++u) {
        const int e = e0 + u * 32 + lane;
        jj[u] = 0;
        ok[u] = false;
        if (e < kk) {
          const int s = e / k, t = e - s * k;
          const uint32_t a = nbid[s];
          if (a != kNoId) {
            jj[u] = id_in[(size_t)a * k + t] & kIdMask;
            const bool jf = flags_in ? ((flags_in[(size_t)a * kw + (t >> 5)] >> (t & 31)) & 1u) : true;
            ok[u] = (nbfl[s] != 0 || jf) && (int64_t)jj[u] < n;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kGatherUnroll; ++u) {
        const bool cand = ok[u] && hash_insert(H, hbits, (int32_t)jj[u]);
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cand);
        if (cand) Q[qn + __popc(bal & lt_mask)] = jj[u];
        qn += __popc(bal);
      }
    }
    __syncwarp();

    // keys of the candidates, 32 per batch, one row slice of kSliceBytes per
    // stage; rows are kRowStride apart, so lane r's 16-byte loads of unit q
    // (address r * 272 + 16 q) fall in distinct bank groups within each
    // 8-lane phase and the unit offsets are compile-time constants
    const int stages = ((qn + 31) >> 5) * nch;
    const int half = lane >> 4, c16 = lane & 15;
    // stage t: rows 32 b .. of the candidates, dims c * kCH .. of each, into buffer t mod NBUF
    auto stage_rows = [&](int t) {
      const int b = t / nch, c = t - b * nch;
      const int m = min(32, qn - 32 * b);
      const int dim = c * kCH + kEPU * c16;
      const bool ok = dim < ldr;
      unsigned char* buf = (NBUF == 2 && (t & 1)) ? rows1 : rows0;
      for (int r = half; r < m; r += 2) {
        const uint32_t jid = Q[32 * b + r];
        cp_async16(buf + r * kRowStride + c16 * 16, X + (size_t)jid * ldr + (ok ? dim : 0), ok ? 16 : 0);
      }
      cp_async_commit();
    };
    float total = 0.f, part = 0.f;
    if (NBUF == 2 && stages > 0) stage_rows(0);
    for (int t = 0; t < stages; ++t) {
      const int b = t / nch, c = t - b * nch;
      const int m = min(32, qn - 32 * b);
      const int cd = c * kCH;
      if (NBUF == 2) {
        if (t + 1 < stages) {
          stage_rows(t + 1);  // its buffer was last read in stage t - 1, before that stage's closing syncwarp
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
      } else {
        stage_rows(t);
        cp_async_wait<0>();
      }
      __syncwarp();
      const unsigned char* rows = (NBUF == 2 && (t & 1)) ? rows1 : rows0;
      if (lane < m) {
        const unsigned char* myrow = rows + lane * kRowStride;
        const int nu = (min(kCH, d - cd) + kEPU - 1) / kEPU;  // 16-byte units holding dims
        const float* qx = xq + cd;
#pragma unroll
        for (int q = 0; q < kCH / kEPU; ++q) {
          if (q < nu) {
            const uint4 raw = *reinterpret_cast<const uint4*>(myrow + q * 16);
            if (HALF) {
              const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 cv = __half22float2(h2[e]);
                part = acc_step<METRIC>(qx[kEPU * q + 2 * e], cv.x, part);
                part = acc_step<METRIC>(qx[kEPU * q + 2 * e + 1], cv.y, part);
              }
            } else {
              const float4 cv = *reinterpret_cast<const float4*>(&raw);
              const float4 qv = *reinterpret_cast<const float4*>(qx + kEPU * q);
              part = acc_step<METRIC>(qv.x, cv.x, part);
              part = acc_step<METRIC>(qv.y, cv.y, part);
              part = acc_step<METRIC>(qv.z, cv.z, part);
              part = acc_step<METRIC>(qv.w, cv.w, part);
            }
          }
        }
        if (((cd + kCH) & 255) == 0 || cd + kCH >= d) {
          total = __fadd_rn(total, part);
          part = 0.f;
        }
      }
      __syncwarp();  // the buffer is refilled by the next stage
      if (c == nch - 1) {
        const int32_t cj = lane < m ? (int32_t)Q[32 * b + lane] : 0;
        float key = total;
        if (METRIC == KNN_METRIC_COSINE) key = lane < m ? cosine_key(total, ni, norms[cj]) : kInf;
        float tk;
        uint32_t ti;
        warp_list_get(L, k - 1, tk, ti);
        const bool pass = lane < m && cand_less(key, (uint32_t)cj, tk, ti);
        if (lane == 0) evaluated += (unsigned long long)m;
        if (__any_sync(0xFFFFFFFFu, pass))
          warp_list_insert(L, pass ? key : kInf, pass ? ((uint32_t)cj | 0x80000000u) : kNoId);
        total = 0.f;
        part = 0.f;
      }
    }

#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      if (e < k) {
        key_out[(size_t)i * k + e] = L.key[r];
        id_out[(size_t)i * k + e] = L.id[r] & kIdMask;
      }
      const uint32_t fl = __ballot_sync(0xFFFFFFFFu, e < k && (L.id[r] >> 31));
      if (lane == 0 && r < kw) flags_out[(size_t)i * kw + r] = fl;
    }
    __syncwarp();
  }
  if (cand_counter && lane == 0 && evaluated) atomicAdd(cand_counter, evaluated);
}

// ------------------------------------------------------- filtered candidates --
// Most candidates of a step lose to the list's last entry, and the exact key must
// be summed in one fixed order by one lane.  So every candidate is first bounded
// from below with 16-bit rows, summed in whatever order is fastest, and only
// those that might enter get their exact key.
//
// 16-bit rows: FP16 of s * x (EUCLIDEAN, TAXICAB; s the power of two that brings
// the largest |x| of all rows into [2^14, 2^15)) or of the unit row (COSINE),
// with the row's rounding error delta >= |s x - h| (L2 norm; L1 for TAXICAB).
// The triangle inequality bounds the distance of the rows by that of the
// 16-bit rows and both deltas; g covers FP32 rounding of either sum.  A row whose
// values defeat the bound (infinite, or a norm whose square leaves the FP32
// range) has delta = inf and is never rejected.
constexpr float kDeltaUp = 1.0f + 1.0f / 1024.0f;  // delta is itself computed in FP32

// Largest |x| over the rows (non-negative floats order as their bit patterns).
__global__ void __launch_bounds__(256) k_max_abs(const float4* __restrict__ X, int64_t count,
                                                      unsigned int* __restrict__ out) {
  float m = 0.f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 v = __ldg(X + i);
    m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
  }
  m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// The scale s for the largest |x| m (1 when m is 0 or not finite).
__device__ __forceinline__ float prop_scale(float m) {
  if (!(m > 0.f && m < __int_as_float(0x7F800000))) return 1.f;
  int e;
  frexpf(m, &e);  // m in [2^(e-1), 2^e)
  return ldexpf(1.f, max(-126, min(126, 15 - e)));
}

// One warp per row: the 16-bit row [ldh] (zero padded) and its delta.
template <int METRIC>
__global__ void __launch_bounds__(256) k_prop_rows(const float* __restrict__ X, int64_t n, int d, int dpad, int ldh,
                                                   const unsigned int* __restrict__ maxabs,
                                                   const float* __restrict__ norms, __half* __restrict__ H,
                                                   float* __restrict__ delta) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  float scale = 1.f;
  bool usable = true;
  if (METRIC == KNN_METRIC_COSINE) {
    const float nr = norms[row];
    usable = nr == 0.f || (nr > 8.67361738e-19f && nr < 1.15292150e18f);  // 2^-60, 2^60
    scale = nr > 0.f ? __frcp_rn(nr) : 0.f;
  } else {
    scale = prop_scale(__uint_as_float(*maxabs));
  }
  float err = 0.f;
  for (int c = lane; c < ldh; c += 32) {
    const float v = c < d ? __fmul_rn(X[(size_t)row * dpad + c], scale) : 0.f;
    const __half h = __float2half_rn(v);
    H[(size_t)row * ldh + c] = h;
    const float e = __fsub_rn(v, __half2float(h));
    err = METRIC == KNN_METRIC_TAXICAB ? __fadd_rn(err, fabsf(e)) : __fmaf_rn(e, e, err);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) err = __fadd_rn(err, __shfl_xor_sync(0xFFFFFFFFu, err, off));
  if (METRIC != KNN_METRIC_TAXICAB) err = __fsqrt_rn(err);
  // NaN (infinite values) and unusable rows: never rejected
  if (lane == 0) delta[row] = usable && err < __int_as_float(0x7F800000) ? err * kDeltaUp : __int_as_float(0x7F800000);
}

// Bounds of a pair from the sum `a` over its 16-bit rows (dsum: both deltas), in
// units of s * distance (EUCLIDEAN, TAXICAB) or key (COSINE): lo exceeds a list
// bound hi only where the pair's FP32 key exceeds the bounding one's.  Past `top`
// the FP32 key may overflow to +inf, which ties by id: hi is no bound there, nor
// when it is NaN.  COSINE: errors of unit rows add, delta^2 < delta / 1024.
struct PairBounds {
  float lo, hi;
};
template <int METRIC>
__device__ __forceinline__ PairBounds pair_bounds(float a, float dsum, float g, float top) {
  PairBounds b;
  if (METRIC == KNN_METRIC_COSINE) {
    const float e = dsum * (1.f + 0.0009765625f) + 4.f * g;
    b.lo = (1.f - a) - e;
    b.hi = (1.f - a) + e;
  } else {
    const float r = METRIC == KNN_METRIC_EUCLIDEAN ? __fsqrt_rn(a) : a;
    b.lo = r * (1.f - g) - dsum;
    b.hi = (r + dsum) * (1.f + g);
  }
  b.hi = b.hi < top ? b.hi : __int_as_float(0x7F800000);
  return b;
}
// An exact key in the same units.
template <int METRIC>
__device__ __forceinline__ float key_bound(float key, float scale, float g) {
  if (METRIC == KNN_METRIC_EUCLIDEAN) return scale * (__fsqrt_rn(key) * (1.f + g));
  if (METRIC == KNN_METRIC_TAXICAB) return scale * (key * (1.f + g));
  return key;
}

// Lane-wise lists of floats: ascending sort, and the 32 smallest of two sorted.
__device__ __forceinline__ float warp_sort32_f(float v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int m = size >> 1; m >= 1; m >>= 1) {
      const float o = __shfl_xor_sync(0xFFFFFFFFu, v, m);
      v = (((lane & size) == 0) == ((lane & m) == 0)) ? fminf(v, o) : fmaxf(v, o);
    }
  return v;
}
__device__ __forceinline__ float warp_merge_lower_f(float a, float b) {
  const int lane = threadIdx.x & 31;
  a = fminf(a, __shfl_sync(0xFFFFFFFFu, b, 31 - lane));
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) {
    const float o = __shfl_xor_sync(0xFFFFFFFFu, a, m);
    a = (lane & m) == 0 ? fminf(a, o) : fmaxf(a, o);
  }
  return a;
}

inline size_t filt_region0_bytes(int k, int d) {
  // hash set (then the candidates' lower bounds: it holds twice k * k entries) or the exact keys' rows and query
  return std::max((size_t)4 << prop_hash_bits(k), (size_t)32 * kFiltPitch + (size_t)4 * round_up(d, 32));
}
inline size_t filt_warp_bytes(int k, int d) {
  const size_t b = filt_region0_bytes(k, d) + (size_t)4 * round_up(k * k, 32) + (size_t)4 * round_up(k, 32) +
                   (size_t)4 * round_up(k * ((k + 31) / 32), 32);
  return (b + 15) & ~(size_t)15;
}

// One warp per point, as k_propagate, with the filter: lanes in groups of
// 2^glog read one candidate's 16-bit row each (8 elements a lane and step, NS
// steps), the query's share of dims in registers, kInFlight candidates' loads in
// flight per group.  No row passes through shared memory before the few exact keys, so
// shared memory holds little more than the hash set and more warps share an SM.
//
// What bounds it: at d = 784 the candidates' row reads, which come from L2 at about
// 5 TB/s with this kernel as with k_propagate, so halving the bytes nearly halves
// the time (200,000 x 784, k=30, L1, four steps: 285 -> 141 ms).  Up to 256 dims
// it is latency: four blocks of eight warps per SM (64 registers) measured faster
// than three or two with more loads in flight, and than five (500,000 x 128 integer
// rows, k=16, five steps: 34.1 ms before; 13.7, 15.7, 21.6 and 15.2 ms; 200,000 x
// 37 COSINE, k=21, two steps: 12.2 -> 4.2 ms).  The registers of NS = 4 want two.
constexpr int filt_blocks(int ns) { return ns == 1 ? 4 : ns == 2 ? 3 : 2; }
template <int METRIC, int KPL, int NS>
__global__ void __launch_bounds__(kPropMaxWarps * 32, filt_blocks(NS)) k_propagate_filtered(
    const float* __restrict__ X, int dpad, const __half* __restrict__ H, int ldh, const float* __restrict__ delta,
    const unsigned int* __restrict__ maxabs, float g, int glog, int64_t n, int64_t r0, int64_t cnt, int d, int k, int kw,
    int hbits, size_t warp_bytes, size_t region0, const float* __restrict__ norms, const int32_t* __restrict__ order,
    const float* __restrict__ key_in, const uint32_t* __restrict__ id_in, const uint32_t* __restrict__ flags_in,
    float* __restrict__ key_out, uint32_t* __restrict__ id_out, uint32_t* __restrict__ flags_out,
    unsigned long long* __restrict__ cand_counter) {
  constexpr int kInFlight = NS == 4 ? 2 : 4;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* base = smem + (size_t)warp * warp_bytes;
  const int hsize = 1 << hbits;
  const int kk = k * k;
  const int kr = (k + 31) & ~31;
  int32_t* Hs = reinterpret_cast<int32_t*>(base);                         // hash set, then:
  unsigned char* rows = base;                                             // [32][kFiltPitch] exact row slices
  float* xq = reinterpret_cast<float*>(base + (size_t)32 * kFiltPitch);  // the query row
  uint32_t* Q = reinterpret_cast<uint32_t*>(base + region0);
  uint32_t* nbid = Q + ((kk + 31) & ~31);
  uint32_t* nbmask = nbid + kr;  // [k][kw] entries of each neighbour's list that may be new candidates
  const float kInf = __int_as_float(0x7F800000);
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int gl = lane & ((1 << glog) - 1), sub = lane >> glog, per = 32 >> glog;  // candidates per step
  const int kp = min(32, 1 << (32 - __clz(max(k - 1, 1)))), lists = 32 / kp, sl = lane / kp;
  const float scale = METRIC == KNN_METRIC_COSINE ? 1.f : prop_scale(__uint_as_float(*maxabs));
  // EUCLIDEAN: squares may underflow where the scaled ones do not (d 2^-138)
  const float under = METRIC == KNN_METRIC_EUCLIDEAN ? scale * __fsqrt_rn((float)d * 2.8698593e-42f) * 1.01f : 0.f;
  // distances whose key stays finite in FP32 (sqrt of the largest float, or itself, with a margin)
  const float top = METRIC == KNN_METRIC_EUCLIDEAN ? scale * 1.8e19f : METRIC == KNN_METRIC_TAXICAB ? scale * 3.3e38f : kInf;
  unsigned long long evaluated = 0;

  const int wpb = blockDim.x >> 5;
  const int64_t nwarps = (int64_t)gridDim.x * wpb;
  for (int64_t w = (int64_t)blockIdx.x * wpb + warp; w < cnt; w += nwarps) {
    const int32_t i = order ? order[r0 + w] : (int32_t)(r0 + w);
    WarpList<KPL> L;
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      uint32_t nid = kNoId, nfl = 0;
      L.key[r] = kInf;
      L.id[r] = kNoId;
      if (e < k) {
        // an id outside [0, n) is an empty entry: kept out of the list and never followed
        const uint32_t u = id_in[(size_t)i * k + e] & kIdMask;
        if (u < (uint64_t)n) {
          L.key[r] = key_in[(size_t)i * k + e];
          L.id[r] = u;
          nid = u;
        }
        nfl = flags_in ? ((flags_in[(size_t)i * kw + r] >> lane) & 1u) : 1u;
      }
      if (e < k) {
        nbid[e] = nid;
        // a listed-before neighbour contributes only the entries new to its list
        for (int x = 0; x < kw; ++x)
          nbmask[e * kw + x] = nid == kNoId ? 0u : (nfl ? 0xFFFFFFFFu : flags_in[(size_t)nid * kw + x]);
      }
    }
    for (int s = lane; s < hsize / 4; s += 32) reinterpret_cast<int4*>(Hs)[s] = make_int4(-1, -1, -1, -1);
    // the lane's dims of the query's 16-bit row
    float q[NS][8];
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      const int e = ((t << glog) + gl) * 8;
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (e < ldh) raw = __ldg(reinterpret_cast<const uint4*>(H + (size_t)i * ldh + e));
      const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 f = __half22float2(h2[p]);
        q[t][2 * p] = f.x;
        q[t][2 * p + 1] = f.y;
      }
    }
    const float dq = delta[i];
    __syncwarp();
    if (lane == 0) hash_insert(Hs, hbits, i);
#pragma unroll
    for (int r = 0; r < KPL; ++r)
      if (r * 32 + lane < k && L.id[r] != kNoId) hash_insert(Hs, hbits, (int32_t)L.id[r]);
    __syncwarp();
    const float ni = (METRIC == KNN_METRIC_COSINE) ? norms[i] : 0.f;

    // candidates: a group of kp lanes (k rounded up to a power of two, at most 32)
    // reads one neighbour's list, kGatherUnroll lists per group in flight
    int qn = 0;
    for (int s0 = 0; s0 < k; s0 += kGatherUnroll * lists) {
      for (int t = lane & (kp - 1); t < kr; t += 32) {  // one round up to k = 32 (t >= k: none)
        uint32_t jj[kGatherUnroll];
#pragma unroll
        for (int u = 0; u < kGatherUnroll; ++u) {
          const int s = s0 + u * lists + sl;
          jj[u] = kNoId;
          if (s < k && t < k && ((nbmask[s * kw + (t >> 5)] >> (t & 31)) & 1u)) jj[u] = id_in[(size_t)nbid[s] * k + t] & kIdMask;
        }
#pragma unroll
        for (int u = 0; u < kGatherUnroll; ++u) {
          const bool cand = jj[u] < (uint64_t)n && hash_insert(Hs, hbits, (int32_t)jj[u]);
          const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cand);
          if (cand) Q[qn + __popc(bal & lt_mask)] = jj[u];
          qn += __popc(bal);
        }
      }
    }
    __syncwarp();
    if (lane == 0) evaluated += (unsigned long long)qn;

    // the filter, 32 candidates at a time: lane c ends up with candidate c's sum.
    // Their lower bounds go over the hash set, and up to k = 32 the smallest upper
    // bounds (the list's own keys first) are kept: the k-th of them bounds the
    // k-th key after this step, which lets about k candidates through instead of
    // all that beat the present list.
    float* lo_b = reinterpret_cast<float*>(base);
    float best = key_bound<METRIC>(L.key[0], scale, g);  // ascending over the lanes (KPL = 1)
    if (!(best < kInf)) best = kInf;
    for (int b0 = 0; b0 < qn; b0 += 32) {
      const int m = min(32, qn - b0);
      const int steps = (m + per - 1) / per;
      const uint32_t cj = lane < m ? Q[b0 + lane] : 0u;
      const float dj = lane < m ? __ldg(delta + cj) : 0.f;
      float mine = 0.f;
      for (int s0 = 0; s0 < steps; s0 += kInFlight) {
        uint4 raw[kInFlight][NS];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const int c = (s0 + u) * per + sub;
          const uint32_t jid = __shfl_sync(0xFFFFFFFFu, cj, c & 31);
          const __half* row = H + (size_t)jid * ldh;
#pragma unroll
          for (int t = 0; t < NS; ++t) {
            const int e = ((t << glog) + gl) * 8;
            raw[u][t] = make_uint4(0u, 0u, 0u, 0u);
            if (c < m && e < ldh) raw[u][t] = __ldg(reinterpret_cast<const uint4*>(row + e));
          }
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          if (s0 + u < steps) {  // warp-uniform
            float s1 = 0.f, s2 = 0.f;
#pragma unroll
            for (int t = 0; t < NS; ++t) {
              const __half2* h2 = reinterpret_cast<const __half2*>(&raw[u][t]);
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                const float2 f = __half22float2(h2[p]);
                s1 = acc_step<METRIC>(q[t][2 * p], f.x, s1);
                s2 = acc_step<METRIC>(q[t][2 * p + 1], f.y, s2);
              }
            }
            float sum = s1 + s2;
            for (int off = (1 << glog) >> 1; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
            const float v = __shfl_sync(0xFFFFFFFFu, sum, (lane & (per - 1)) << glog);
            if (lane / per == s0 + u) mine = v;
          }
        }
      }
      const PairBounds bounds = pair_bounds<METRIC>(mine, dq + dj, g, top);
      lo_b[b0 + lane] = bounds.lo;
      if (KPL == 1) best = warp_merge_lower_f(best, warp_sort32_f(lane < m ? bounds.hi : kInf));
    }
    __syncwarp();
    float tk;
    uint32_t ti;
    warp_list_get(L, k - 1, tk, ti);
    float limit = key_bound<METRIC>(tk, scale, g);
    if (KPL == 1) limit = fminf(limit, __shfl_sync(0xFFFFFFFFu, best, k - 1));
    limit = limit * (METRIC == KNN_METRIC_COSINE ? 1.f : 1.f + g) + under;
    // candidates that may enter, compacted to the front of Q
    int qs = 0;
    for (int b0 = 0; b0 < qn; b0 += 32) {
      const uint32_t cj = Q[b0 + lane < qn ? b0 + lane : 0];
      const bool keep = b0 + lane < qn && !(lo_b[b0 + lane] > limit);
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, keep);
      if (keep) Q[qs + __popc(bal & lt_mask)] = cj;  // qs <= b0: below the entries still to read
      qs += __popc(bal);
    }
    __syncwarp();

    // exact keys of the kept candidates, one lane per candidate in the
    // reference's order, 32-dim slices of the 32 rows at a time (the hash set is done with)
    if (qs > 0)
      for (int c = lane; c < ((d + 31) & ~31); c += 32) xq[c] = c < d ? X[(size_t)i * dpad + c] : 0.f;
    for (int b0 = 0; b0 < qs; b0 += 32) {
      const int m = min(32, qs - b0);
      const uint32_t cj = lane < m ? Q[b0 + lane] : 0u;
      // fewer rows take wider slices of the same buffer, so fewer waits
      const int wlog = m <= 8 ? 7 : m <= 16 ? 6 : 5, width = 1 << wlog, pitch = 4 * width + 16;
      const int ulog = wlog - 2, r1 = lane >> ulog, c1 = lane & ((1 << ulog) - 1), rstep = 32 >> ulog;
      float total = 0.f, part = 0.f;
      for (int cd = 0; cd < d; cd += width) {
        const int dim = cd + 4 * c1;
        for (int r = r1; r < m; r += rstep) {
          const uint32_t jid = Q[b0 + r];
          cp_async16(rows + r * pitch + c1 * 16, X + (size_t)jid * dpad + (dim < dpad ? dim : 0), dim < dpad ? 16 : 0);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        if (lane < m) {
          const float* myrow = reinterpret_cast<const float*>(rows + lane * pitch);
          const int nu = (min(width, d - cd) + 3) / 4;
          const float* qx = xq + cd;
#pragma unroll 8
          for (int u = 0; u < nu; ++u) {
            const float4 cv = *reinterpret_cast<const float4*>(myrow + 4 * u);
            const float4 qv = *reinterpret_cast<const float4*>(qx + 4 * u);
            part = acc_step<METRIC>(qv.x, cv.x, part);
            part = acc_step<METRIC>(qv.y, cv.y, part);
            part = acc_step<METRIC>(qv.z, cv.z, part);
            part = acc_step<METRIC>(qv.w, cv.w, part);
          }
          if (((cd + width) & 255) == 0 || cd + width >= d) {
            total = __fadd_rn(total, part);
            part = 0.f;
          }
        }
        __syncwarp();  // the rows are refilled by the next slice
      }
      float key = total;
      if (METRIC == KNN_METRIC_COSINE) key = lane < m ? cosine_key(total, ni, norms[cj]) : kInf;
      warp_list_get(L, k - 1, tk, ti);
      const bool pass = lane < m && cand_less(key, cj, tk, ti);
      if (__any_sync(0xFFFFFFFFu, pass))
        warp_list_insert(L, pass ? key : kInf, pass ? (cj | 0x80000000u) : kNoId);
    }

#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      if (e < k) {
        key_out[(size_t)i * k + e] = L.key[r];
        id_out[(size_t)i * k + e] = L.id[r] & kIdMask;
      }
      const uint32_t fl = __ballot_sync(0xFFFFFFFFu, e < k && (L.id[r] >> 31));
      if (lane == 0 && r < kw) flags_out[(size_t)i * kw + r] = fl;
    }
    __syncwarp();
  }
  if (cand_counter && lane == 0 && evaluated) atomicAdd(cand_counter, evaluated);
}

template <int METRIC, bool HALF, int NBUF>
static void launch_prop_metric(const PropArgs& a, int kpl, int hbits, size_t wb, int wpb, unsigned grid) {
  const int kw = (a.k + 31) / 32;
  const int64_t r0 = a.r0, cnt = (a.r1 > 0 ? a.r1 : a.n) - a.r0;
  const size_t smem = wb * wpb;
  const void* rows = HALF ? static_cast<const void*>(a.Xh) : static_cast<const void*>(a.X);
  const int ldr = HALF ? a.ldh : a.dpad;
  const size_t region0 = prop_region0_bytes(a.k, NBUF);
#define KNN_PROP_LAUNCH(KP)                                                                                \
  do {                                                                                                     \
    cudaFuncSetAttribute(k_propagate<METRIC, KP, HALF, NBUF>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                         (int)kPropSmemBudget);                                                            \
    k_propagate<METRIC, KP, HALF, NBUF><<<grid, wpb * 32, smem, a.stream>>>(                               \
        rows, ldr, a.n, r0, cnt, a.d, a.k, kw, hbits, wb, region0, a.norms, a.order, a.key_in, a.id_in,    \
        a.flags_in, a.key_out, a.id_out, a.flags_out, a.cand_counter);                                     \
  } while (0)
  if (kpl == 1) KNN_PROP_LAUNCH(1);
  else if (kpl == 2) KNN_PROP_LAUNCH(2);
  else KNN_PROP_LAUNCH(4);
#undef KNN_PROP_LAUNCH
}

template <int METRIC>
static void launch_prop_rows(const PropArgs& a, int kpl, int hbits, size_t wb, int wpb, unsigned grid, int nbuf) {
  if (nbuf == 2) {
    if (a.Xh) launch_prop_metric<METRIC, true, 2>(a, kpl, hbits, wb, wpb, grid);
    else launch_prop_metric<METRIC, false, 2>(a, kpl, hbits, wb, wpb, grid);
  } else {
    if (a.Xh) launch_prop_metric<METRIC, true, 1>(a, kpl, hbits, wb, wpb, grid);
    else launch_prop_metric<METRIC, false, 1>(a, kpl, hbits, wb, wpb, grid);
  }
}

template <int METRIC>
static void launch_filtered(const PropArgs& a, int kpl, int hbits, size_t wb, int wpb, unsigned grid) {
  const int kw = (a.k + 31) / 32;
  const int64_t r0 = a.r0, cnt = (a.r1 > 0 ? a.r1 : a.n) - a.r0;
  const size_t smem = wb * wpb, region0 = filt_region0_bytes(a.k, a.d);
  const int ldh = prop_row_stride(a.d), units = ldh / 8;
  int glog = 0;
  while (glog < 5 && (1 << glog) < units) ++glog;
  const int ns = (units + 31) / 32;
  const float g = (float)(2 * a.d + 64) * 5.9604644775390625e-08f;  // 2^-24
#define KNN_FILT_LAUNCH(KP, NS)                                                                                  \
  do {                                                                                                           \
    cudaFuncSetAttribute(k_propagate_filtered<METRIC, KP, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                         (int)kPropSmemBudget);                                                                  \
    k_propagate_filtered<METRIC, KP, NS><<<grid, wpb * 32, smem, a.stream>>>(                                    \
        a.X, a.dpad, static_cast<const __half*>(a.H), ldh, a.delta, a.maxabs, g, glog, a.n, r0, cnt, a.d, a.k, kw, \
        hbits, wb, region0, a.norms, a.order, a.key_in, a.id_in, a.flags_in, a.key_out, a.id_out, a.flags_out,   \
        a.cand_counter);                                                                                         \
  } while (0)
#define KNN_FILT_NS(KP)                          \
  do {                                           \
    if (ns == 1) KNN_FILT_LAUNCH(KP, 1);         \
    else if (ns == 2) KNN_FILT_LAUNCH(KP, 2);    \
    else KNN_FILT_LAUNCH(KP, 4);                 \
  } while (0)
  if (kpl == 1) KNN_FILT_NS(1);
  else if (kpl == 2) KNN_FILT_NS(2);
  else KNN_FILT_NS(4);
#undef KNN_FILT_NS
#undef KNN_FILT_LAUNCH
}

// Blocks per SM of k_propagate with its warps per block (one row-slice buffer).
static int exact_blocks(int k, int d, int* wpb) {
  const size_t wb = prop_warp_bytes(k, d, 1);
  *wpb = (int)std::min<size_t>(kPropMaxWarps, kPropSmemBudget / wb);
  return *wpb < 1 ? 0 : std::max(1, (int)((220 * 1024) / (wb * *wpb)));
}

bool prop_filter_applies(int k, int d) {
  return d <= kFiltMaxDim && filt_warp_bytes(k, d) <= kPropSmemBudget;
}

// Whether the filter is the faster one.  Where k_propagate keeps two blocks of eight warps per
// SM (lists up to 15, fewer from 576 dims on), it is not always: it reads FP16 input at
// half the bytes too, COSINE keys cost it one instruction per dim, and the filter's lanes
// read power-of-two widths (`idle` = width over dims).  Two steps, 100,000 points, 64 clusters,
// filter against exact, EUCLIDEAN / COSINE, k = 8: 136 dims 1.14 / 1.18, 192 1.10 / 1.18, 208
// 0.96 / 1.03, 256 0.95 / 1.05, 300 1.18 / 1.31, 384 1.05 / 1.21, 448 0.98 / 1.15, 512 0.91 / 1.10,
// 520 1.27 / 1.50, 784 1.00 / 1.14, 900 0.89 / 1.24, 1,000 0.50 / 0.82 (one block); FP16 input
// 96 dims 0.98, 136 1.24, 256 1.17, 520 1.61.  k = 4: 136 0.99 / 1.01, 340 0.95 / 1.09, 520
// 1.07 / 1.27, FP16 136 0.99, 340 1.16.  Tiny rows
// and lists leave nothing to reject: k = 5, 8 dims 1.44 / 1.20, 16 dims 1.07 / 0.91; k = 3, 40 dims
// 1.43 / 1.29, 72 0.92 / 0.85.  One block per SM: 0.29 to 0.99.
bool prop_filter_pays(int k, int d, int metric, bool half) {
  if ((k <= 5 && d <= 8) || (k <= 3 && d <= 40)) return false;
  int wpb;
  const bool cosine = metric == KNN_METRIC_COSINE;
  const int shortest = d > 256 && (half || cosine) ? 4 : 5;  // shorter lists: the filter
  if (d <= 128 || k < shortest || exact_blocks(k, d, &wpb) < 2 || wpb < kPropMaxWarps) return true;
  if (half) return false;
  int width = 256;
  while (width < d) width *= 2;
  const double idle = (double)width / d;
  if (cosine) return idle < (d <= 256 ? 1.33 : 1.12);
  return d <= 256 ? idle < 1.33 || k < 6 : idle < 1.45;
}

void launch_max_abs(const float* X, int64_t n, int dpad, unsigned int* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, sizeof(unsigned int), st);
  const int64_t quads = n * (int64_t)(dpad / 4);
  k_max_abs<<<(unsigned)std::min<int64_t>((quads + 255) / 256, 148 * 8), 256, 0, st>>>(reinterpret_cast<const float4*>(X),
                                                                                       quads, out);
}

int prop_prepare(const PropPrep& a, LaunchLog& log) {
  const int ldh = prop_row_stride(a.d);
  __half* H = static_cast<__half*>(a.H);
  if (a.metric != KNN_METRIC_COSINE) {
    launch_max_abs(a.X, a.n, a.dpad, a.maxabs, a.stream);
    log.add();
  }
  const unsigned grid = (unsigned)((a.n + 7) / 8);
  if (a.metric == KNN_METRIC_EUCLIDEAN)
    k_prop_rows<KNN_METRIC_EUCLIDEAN><<<grid, 256, 0, a.stream>>>(a.X, a.n, a.d, a.dpad, ldh, a.maxabs, a.norms, H, a.delta);
  else if (a.metric == KNN_METRIC_TAXICAB)
    k_prop_rows<KNN_METRIC_TAXICAB><<<grid, 256, 0, a.stream>>>(a.X, a.n, a.d, a.dpad, ldh, a.maxabs, a.norms, H, a.delta);
  else
    k_prop_rows<KNN_METRIC_COSINE><<<grid, 256, 0, a.stream>>>(a.X, a.n, a.d, a.dpad, ldh, a.maxabs, a.norms, H, a.delta);
  log.add();
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

int propagate_step(const PropArgs& a, LaunchLog& log) {
  const int kpl = kpl_for(a.k);
  const int hbits = prop_hash_bits(a.k);
  if (a.H && prop_filter_applies(a.k, a.d)) {
    const size_t fb = filt_warp_bytes(a.k, a.d);
    int wpb = (int)std::min<size_t>(kPropMaxWarps, kPropSmemBudget / fb);
    if (a.warps > 0 && a.warps < wpb) wpb = a.warps;
    const int64_t cnt = (a.r1 > 0 ? a.r1 : a.n) - a.r0;
    if (cnt <= 0) return KNN_OK;
    // several blocks' worth of points per resident block: points differ in
    // their candidates, and blocks that end early make room
    const unsigned grid = (unsigned)std::min<int64_t>((cnt + wpb - 1) / wpb, 148 * 64);
    if (a.metric == KNN_METRIC_EUCLIDEAN) launch_filtered<KNN_METRIC_EUCLIDEAN>(a, kpl, hbits, fb, wpb, grid);
    else if (a.metric == KNN_METRIC_TAXICAB) launch_filtered<KNN_METRIC_TAXICAB>(a, kpl, hbits, fb, wpb, grid);
    else launch_filtered<KNN_METRIC_COSINE>(a, kpl, hbits, fb, wpb, grid);
    log.add();
    return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
  }
  size_t wb = prop_warp_bytes(a.k, a.d, 1);
  int wpb;
  if (exact_blocks(a.k, a.d, &wpb) < 1) return KNN_ERR_UNSUPPORTED;
  if (a.warps > 0 && a.warps < wpb) wpb = a.warps;  // a tuned block size (results identical)
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per_sm = (int)((220 * 1024) / (wb * wpb));
  if (per_sm < 1) per_sm = 1;
  // a second row-slice buffer where it leaves the warps per SM as they are
  // (the results do not depend on it)
  int nbuf = 1;
  const size_t wb2 = prop_warp_bytes(a.k, a.d, 2);
  if (wb2 * wpb <= kPropSmemBudget && (int)((220 * 1024) / (wb2 * wpb)) >= per_sm) {
    nbuf = 2;
    wb = wb2;
  }
  const int64_t cnt = (a.r1 > 0 ? a.r1 : a.n) - a.r0;
  if (cnt <= 0) return KNN_OK;
  const int64_t want = (cnt + wpb - 1) / wpb;
  const int64_t cap = (int64_t)sms * per_sm;
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  if (a.metric == KNN_METRIC_EUCLIDEAN) launch_prop_rows<KNN_METRIC_EUCLIDEAN>(a, kpl, hbits, wb, wpb, grid, nbuf);
  else if (a.metric == KNN_METRIC_TAXICAB) launch_prop_rows<KNN_METRIC_TAXICAB>(a, kpl, hbits, wb, wpb, grid, nbuf);
  else launch_prop_rows<KNN_METRIC_COSINE>(a, kpl, hbits, wb, wpb, grid, nbuf);
  log.add();
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

}  // namespace knn
