// Exact k-NN in FP64 on the GPU: the yardstick of recall and distance error.
// No counterpart in the reference (which never checks its own output; its
// VALIDATION file is written unconditionally, euclideandistancematrixgpu.cu:2967-2971).
//
// Arithmetic matches a plain sequential double loop without contraction:
//   L2:  sqrt(sum (a-b)^2),  L1: sum |a-b|,  COS: 1 - sum ab / (sqrt(sum a^2) sqrt(sum b^2))
// and ties break by index, so the result equals a CPU double-precision brute force.
//
// Layout: a block owns 64 queries and one slice of the points; the 64x64
// distance tile is built by a 4x4 register tile per thread (points staged 8
// dims at a time in shared memory), each warp keeps the sorted k best of 8
// queries in registers.  A second kernel merges the slices.  Long slices go
// through k_exact_filtered, which computes FP64 keys only for the pairs that
// FP32 cannot rule out; k_exact then takes only the blocks it gave up on.
#include "knn_internal.cuh"
#include "knn_kernels.cuh"

namespace knn {

namespace {
constexpr int kET = 64;
constexpr int kEDC = 8;  // keeps the static shared memory under 48 KB
constexpr int kFC = 128;          // k_exact_filtered: candidates per tile,
constexpr int kFD = 16;           // dims per stage,
constexpr int kFHold = 512;       // queued pairs past which a warp empties its queue at once,
constexpr int kFQueue = 8 * kFC + kFHold;  // and a warp's queue: one tile on top of that
constexpr int kFilterMaxDim = 1 << 20;
constexpr uint32_t kRedoMark = 0xFFFFFFFEu;  // first partial id of a block left to k_exact

struct FilterSmem {
  float q[2][kFD][kET + 4];
  float c[2][kFD][kFC + 4];
  uint32_t id[8][kFQueue];
  uint8_t qs[8][kFQueue];
  float cn[kFC];
  float lim[kET];
  int64_t qrow[kET];
};
}  // namespace

__global__ void k_exact_norms(const float* __restrict__ X, int64_t n, int d, int dpad,
                              double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* a = X + (size_t)i * dpad;
  double s = 0.0;
  for (int e = 0; e < d; ++e) s = __dadd_rn(s, __dmul_rn((double)a[e], (double)a[e]));
  out[i] = sqrt(s);
}

template <int METRIC, int KPL>
__global__ void __launch_bounds__(256) k_exact(const float* __restrict__ X, int64_t n, int d,
                                               int dpad, int k, const int64_t* __restrict__ queries,
                                               int64_t nq, const double* __restrict__ norms,
                                               int64_t slice, double* __restrict__ part_dist,
                                               uint32_t* __restrict__ part_idx, bool redo_only) {
  if (redo_only && part_idx[((size_t)blockIdx.y * nq + (int64_t)blockIdx.x * kET) * k] != kRedoMark) return;
  __shared__ double Qs[kEDC][kET + 1];
  __shared__ double Cs[kEDC][kET + 1];
  __shared__ double Ks[kET][kET + 1];
  __shared__ int64_t qrow[kET];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, warp = tid >> 5, lane = tid & 31;
  const int64_t q0 = (int64_t)blockIdx.x * kET;
  const int mq = (int)min((int64_t)kET, nq - q0);
  const int64_t c_begin = (int64_t)blockIdx.y * slice;
  const int64_t c_end = min(n, c_begin + slice);
  const double kInf = __longlong_as_double(0x7FF0000000000000LL);
  if (tid < kET) qrow[tid] = tid < mq ? queries[q0 + tid] : -1;
  __syncthreads();

  WarpList<KPL, double> L[8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      L[s].key[r] = kInf;
      L[s].id[r] = kNoId;
    }

  for (int64_t c0 = c_begin; c0 < c_end; c0 += kET) {
    const int mc = (int)min((int64_t)kET, c_end - c0);
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    for (int cd = 0; cd < d; cd += kEDC) {
      for (int f = tid; f < kET * kEDC; f += 256) {
        const int r = f / kEDC, e = f % kEDC;
        const int dim = cd + e;
        double qv = 0.0, cv = 0.0;
        if (r < mq && dim < d) qv = (double)X[(size_t)qrow[r] * dpad + dim];
        if (r < mc && dim < d) cv = (double)X[(size_t)(c0 + r) * dpad + dim];
        Qs[e][r] = qv;
        Cs[e][r] = cv;
      }
      __syncthreads();
      const int lim = min(kEDC, d - cd);
      for (int e = 0; e < lim; ++e) {
        double qa[4], cb[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) qa[a] = Qs[e][ty * 4 + a];
#pragma unroll
        for (int b = 0; b < 4; ++b) cb[b] = Cs[e][tx * 4 + b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            if (METRIC == KNN_METRIC_EUCLIDEAN) {
              const double t = __dsub_rn(qa[a], cb[b]);
              acc[a][b] = __dadd_rn(acc[a][b], __dmul_rn(t, t));
            } else if (METRIC == KNN_METRIC_TAXICAB) {
              acc[a][b] = __dadd_rn(acc[a][b], fabs(__dsub_rn(qa[a], cb[b])));
            } else {
              acc[a][b] = __dadd_rn(acc[a][b], __dmul_rn(qa[a], cb[b]));
            }
          }
      }
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int qq = ty * 4 + a, cc = tx * 4 + b;
        double v = acc[a][b];
        if (METRIC == KNN_METRIC_EUCLIDEAN) v = sqrt(v);
        if (METRIC == KNN_METRIC_COSINE && qq < mq && cc < mc) {
          const double den = __dmul_rn(norms[qrow[qq]], norms[c0 + cc]);
          v = den == 0.0 ? 1.0 : __dsub_rn(1.0, __ddiv_rn(v, den));
        }
        const bool ok = qq < mq && cc < mc && qrow[qq] != c0 + cc;
        Ks[qq][cc] = ok ? v : kInf;
      }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int qq = warp * 8 + s;
      if (qq >= mq) continue;
      for (int cb = 0; cb < mc; cb += 32) {
        const int c = cb + lane;
        const double ck = c < mc ? Ks[qq][c] : kInf;
        const uint32_t ci = c < mc ? (uint32_t)(c0 + c) : kNoId;
        double tk;
        uint32_t ti;
        warp_list_get(L[s], k - 1, tk, ti);
        const bool pass = ck < kInf && cand_less(ck, ci, tk, ti);
        if (__any_sync(0xFFFFFFFFu, pass)) warp_list_insert(L[s], pass ? ck : kInf, pass ? ci : kNoId);
      }
    }
    __syncthreads();
  }
  // partial result of this slice: [slice][query][k]
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int qq = warp * 8 + s;
    if (qq >= mq) continue;
    const size_t row = ((size_t)blockIdx.y * nq + (q0 + qq)) * k;
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      if (e < k) {
        part_dist[row + e] = L[s].key[r];
        part_idx[row + e] = L[s].id[r];
      }
    }
  }
}

// FP64 key of one pair, the terms added one by one as in k_exact.
template <int METRIC>
__device__ __forceinline__ double exact_step(float qf, float cf, double acc) {
  const double q = (double)qf, c = (double)cf;
  if (METRIC == KNN_METRIC_EUCLIDEAN) {
    const double t = __dsub_rn(q, c);
    return __dadd_rn(acc, __dmul_rn(t, t));
  }
  if (METRIC == KNN_METRIC_TAXICAB) return __dadd_rn(acc, fabs(__dsub_rn(q, c)));
  return __dadd_rn(acc, __dmul_rn(q, c));
}

// What an FP32 sum must exceed (EUCLIDEAN: of squares, TAXICAB) for its pair to
// have an FP64 key above tk, or, times the candidate's norm, fall below (COSINE).
// An FP32 sum of d terms of one sign errs by less than g = (2d + 64) 2^-24 of itself,
// a dot product by g |a| |b|, and every term by 2^-149 more where it underflows.
// Too large sums become +inf and are out only where tk's own square is in range;
// an open list (tk = +inf) and norms whose products could leave FP32's range give a
// limit that nothing passes, and so do NaNs, which no comparison rejects.
template <int METRIC>
__device__ __forceinline__ float exact_limit(double tk, double g, int d, double nq) {
  if (METRIC == KNN_METRIC_COSINE) {
    if (!(tk < 4.0) || !(nq > 9.094947e-13 && nq < 1.152921e18)) return __int_as_float(0xFF800000);
    return __double2float_rd((1.0 - tk - 2.0 * g - 4.76837158203125e-07) * nq);
  }
  const double t = METRIC == KNN_METRIC_EUCLIDEAN ? tk * tk : tk;
  return __double2float_ru(t * (1.0 + 2.0 * g) + (double)d * 2.802596928649634e-45);
}

// k_exact behind an FP32 filter.  A block takes 64 queries x 128 candidates, a
// thread 4 x 8 of them; the threads of a warp hold the keys of exactly the 8 queries
// whose lists the warp keeps, so pairs under the limit go from registers to the
// warp's queue without a barrier.  32 queued pairs at a time get their FP64 keys, one
// lane each in the sequential order, and enter the lists; the limits follow.  Which
// pairs are queued does not change the lists: they hold the k smallest (key, id).
//
// What bounds it: FP32 issue (two instructions per pair and dim, one for COSINE)
// instead of three FP64 instructions at half the rate and their operands' conversions.
// Half of the FP32 peak without the keys; with them, 2000 queries x 200,000 x 128
// on a B200: 23.8 -> 7.8 ms (k=16), 37.1 -> 16.7 (k=40), 18.5 -> 5.9 (k=1); keys
// computed after every tile instead of at growing gaps: 9.8 (k=16).
//
// Data whose k-th keys tie with much of the set (copies of few points) would queue
// most pairs, at about 2.5 times k_exact's cost per pair: a block whose warp has queued a
// third of its pairs, past what open lists take (8 k (1 + ln(candidates / k)) pairs, a first
// tile's 1,024 at most), marks itself for k_exact and ends.  2,000 queries x 100,000 x 64, all
// rows equal, against k_exact alone: k = 16 1.35 with an allowance of 4,096 pairs, 1.00 now, k = 40 1.59
// and 1.2; with 512 + 8 k pairs ordinary data gave up too (k = 100: 37.8 -> 47 ms).
template <int METRIC, int KPL>
__global__ void __launch_bounds__(256, KPL == 1 ? 2 : 1)
    k_exact_filtered(const float* __restrict__ X, int64_t n, int d, int dpad, bool vec, int k,
                     const int64_t* __restrict__ queries, int64_t nq, const double* __restrict__ norms, int64_t slice,
                     double* __restrict__ part_dist, uint32_t* __restrict__ part_idx) {
  extern __shared__ __align__(16) unsigned char exact_smem[];
  FilterSmem& sm = *reinterpret_cast<FilterSmem*>(exact_smem);
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, warp = tid >> 5, lane = tid & 31;
  const int64_t q0 = (int64_t)blockIdx.x * kET;
  const int mq = (int)min((int64_t)kET, nq - q0);
  const int64_t c_begin = (int64_t)blockIdx.y * slice;
  const int64_t c_end = min(n, c_begin + slice);
  const double kInf = __longlong_as_double(0x7FF0000000000000LL);
  const double g = (double)(2 * d + 64) * 5.9604644775390625e-08;
  if (tid < kET) {
    sm.qrow[tid] = queries[q0 + (tid < mq ? tid : 0)];
    sm.lim[tid] = exact_limit<METRIC>(kInf, g, d, 0.0);
  }
  __syncthreads();

  WarpList<KPL, double> L[8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      L[s].key[r] = kInf;
      L[s].id[r] = kNoId;
    }

  // staging: a lane reads 16 bytes of a row, two lanes its 32-byte sector; rows
  // 16 apart in the pitch keep the transposed stores free of bank conflicts
  const int sr = (warp & 3) * 16 + (lane & 15), se = ((warp >> 2) * 2 + (lane >> 4)) * 4;
  const float* const qsrc = X + (size_t)sm.qrow[sr] * dpad;
  auto load4 = [&](const float* row, bool ok, int dim) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!ok) return v;
    if (vec) {
      if (dim < dpad) v = __ldg(reinterpret_cast<const float4*>(row + dim));
    } else {
      if (dim < d) v.x = __ldg(row + dim);
      if (dim + 1 < d) v.y = __ldg(row + dim + 1);
      if (dim + 2 < d) v.z = __ldg(row + dim + 2);
      if (dim + 3 < d) v.w = __ldg(row + dim + 3);
    }
    return v;
  };

  uint32_t* const qid = sm.id[warp];
  uint8_t* const qof = sm.qs[warp];
  int queued = 0;               // pairs waiting in the warp's queue
  int64_t seen = 0, taken = 0;  // pairs filtered and pairs queued so far
  int64_t tile = 0, next_drain = 0;
  const int nch = (d + kFD - 1) / kFD;
  // FP64 keys of the last m <= 32 queued pairs into the lists
  auto drain = [&](int m) {
    const bool on = lane < m;
    const uint32_t ci = on ? qid[queued - m + lane] : 0u;
    const int qs = on ? qof[queued - m + lane] : 0;
    const int64_t qr = sm.qrow[warp * 8 + qs];
    const float* a = X + (size_t)qr * dpad;
    const float* b = X + (size_t)ci * dpad;
    double key = 0.0;
    if (on) {
      int e = 0;
      if (vec) {
#pragma unroll 8
        for (; e + 4 <= d; e += 4) {
          const float4 av = __ldg(reinterpret_cast<const float4*>(a + e));
          const float4 bv = __ldg(reinterpret_cast<const float4*>(b + e));
          key = exact_step<METRIC>(av.x, bv.x, key);
          key = exact_step<METRIC>(av.y, bv.y, key);
          key = exact_step<METRIC>(av.z, bv.z, key);
          key = exact_step<METRIC>(av.w, bv.w, key);
        }
      }
      for (; e < d; ++e) key = exact_step<METRIC>(__ldg(a + e), __ldg(b + e), key);
      if (METRIC == KNN_METRIC_EUCLIDEAN) key = sqrt(key);
      if (METRIC == KNN_METRIC_COSINE) {
        const double den = __dmul_rn(norms[qr], norms[ci]);
        key = den == 0.0 ? 1.0 : __dsub_rn(1.0, __ddiv_rn(key, den));
      }
    }
    queued -= m;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const bool mine = on && qs == s;
      if (!__any_sync(0xFFFFFFFFu, mine)) continue;
      double tk;
      uint32_t ti;
      warp_list_get(L[s], k - 1, tk, ti);
      const bool pass = mine && key < kInf && cand_less(key, ci, tk, ti);
      if (!__any_sync(0xFFFFFFFFu, pass)) continue;
      warp_list_insert(L[s], pass ? key : kInf, pass ? ci : kNoId);
      warp_list_get(L[s], k - 1, tk, ti);
      if (lane == 0)
        sm.lim[warp * 8 + s] = exact_limit<METRIC>(
            tk, g, d, METRIC == KNN_METRIC_COSINE ? norms[sm.qrow[warp * 8 + s]] : 0.0);
    }
    __syncwarp();
  };

  for (int64_t c0 = c_begin; c0 < c_end; c0 += kFC) {
    const int mc = (int)min((int64_t)kFC, c_end - c0);
    float acc[4][8];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) acc[a][b] = 0.f;
    const bool ok0 = sr < mc, ok1 = sr + 64 < mc;
    const float* const csrc0 = X + (size_t)(c0 + (ok0 ? sr : 0)) * dpad;
    const float* const csrc1 = X + (size_t)(c0 + (ok1 ? sr + 64 : 0)) * dpad;
    float4 vq, v0, v1;
    auto fetch = [&](int ch) {
      const int dim = ch * kFD + se;
      vq = load4(qsrc, true, dim);
      v0 = load4(csrc0, ok0, dim);
      v1 = load4(csrc1, ok1, dim);
    };
    auto stage = [&](int buf) {
      const float q4[4] = {vq.x, vq.y, vq.z, vq.w}, a4[4] = {v0.x, v0.y, v0.z, v0.w}, b4[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sm.q[buf][se + u][sr] = q4[u];
        sm.c[buf][se + u][sr] = a4[u];
        sm.c[buf][se + u][sr + 64] = b4[u];
      }
    };
    if (METRIC == KNN_METRIC_COSINE && tid < kFC) {
      // NaN: never rejected
      const double nc = tid < mc ? norms[c0 + tid] : 0.0;
      sm.cn[tid] = nc > 9.094947e-13 && nc < 1.152921e18 ? (float)nc : __int_as_float(0x7FC00000);
    }
    fetch(0);
    stage(0);
    __syncthreads();
    for (int ch = 0; ch < nch; ++ch) {
      const int buf = ch & 1;
      if (ch + 1 < nch) fetch(ch + 1);
#pragma unroll
      for (int e = 0; e < kFD; ++e) {
        const float4 q4 = *reinterpret_cast<const float4*>(&sm.q[buf][e][ty * 4]);
        const float4 a4 = *reinterpret_cast<const float4*>(&sm.c[buf][e][tx * 4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&sm.c[buf][e][64 + tx * 4]);
        const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
        const float cv[8] = {a4.x, a4.y, a4.z, a4.w, b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            if (METRIC == KNN_METRIC_COSINE) {
              acc[a][b] = __fmaf_rn(qv[a], cv[b], acc[a][b]);
            } else {
              const float t = __fsub_rn(qv[a], cv[b]);
              acc[a][b] = METRIC == KNN_METRIC_EUCLIDEAN ? __fmaf_rn(t, t, acc[a][b]) : __fadd_rn(acc[a][b], fabsf(t));
            }
          }
      }
      if (ch + 1 < nch) stage(buf ^ 1);
      __syncthreads();
    }

    // Pairs under the limit are queued.  The keys take long (a serial chain of d adds
    // per lane), and a warp at them holds its block at the next barrier, so all warps
    // empty their queues after the same tiles, at gaps that grow with the tiles seen,
    // as the pairs per tile fall.  The first tile goes in four steps of 32 candidates, each
    // with the limits of the last.
    const bool open = tile == 0, empty = tile >= next_drain;
    if (empty) next_drain = tile + 1 + tile / 4;
    ++tile;
    for (int step = 0; step < (open ? 4 : 1); ++step) {
      uint32_t mask = 0;  // bit 8a + b
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float lim = sm.lim[ty * 4 + a];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const float v = acc[a][b];
          const int cc = (b >> 2) * 64 + tx * 4 + (b & 3);
          const bool out = METRIC == KNN_METRIC_COSINE ? v < lim * sm.cn[cc] : v > lim;
          if (!out && cc < mc) mask |= 1u << (8 * a + b);
        }
        if (ty * 4 + a >= mq) mask &= ~(0xFFu << (8 * a));
        const int64_t self = sm.qrow[ty * 4 + a] - c0;  // the query itself
        if (self >= 0 && self < kFC && (int)(self & 63) >> 2 == tx)
          mask &= ~(1u << (8 * a + (int)(self >> 6) * 4 + (int)(self & 3)));
      }
      if (open) mask &= 0x03030303u << (2 * step);
      if (__any_sync(0xFFFFFFFFu, mask != 0)) {
        const int cnt = __popc(mask);
        int at = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int o = __shfl_up_sync(0xFFFFFFFFu, at, off);
          if (lane >= off) at += o;
        }
        const int total = __shfl_sync(0xFFFFFFFFu, at, 31);
        at += queued - cnt;
        while (mask) {
          const int bit = __ffs(mask) - 1, a = bit >> 3, b = bit & 7;
          mask &= mask - 1;
          qid[at] = (uint32_t)(c0 + (b >> 2) * 64 + tx * 4 + (b & 3));
          qof[at] = (uint8_t)((ty & 1) * 4 + a);
          ++at;
        }
        queued += total;
        taken += total;
        __syncwarp();
      }
      if (empty || queued >= kFHold)
        while (queued > 0) drain(min(queued, 32));
    }
    seen += 8 * kFC;
    // every warp sees the same verdict; the barrier also keeps the next tile's
    // norms from overwriting those that a late warp still reads
    if (__syncthreads_or(taken > (KPL <= 2 ? 512 : 1024) + 16 * k + seen / 3)) {
      if (tid == 0) part_idx[((size_t)blockIdx.y * nq + q0) * k] = kRedoMark;
      return;
    }
  }
  while (queued > 0) drain(min(queued, 32));
  // partial result of this slice: [slice][query][k]
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int qq = warp * 8 + s;
    if (qq >= mq) continue;
    const size_t row = ((size_t)blockIdx.y * nq + (q0 + qq)) * k;
#pragma unroll
    for (int r = 0; r < KPL; ++r) {
      const int e = r * 32 + lane;
      if (e < k) {
        part_dist[row + e] = L[s].key[r];
        part_idx[row + e] = L[s].id[r];
      }
    }
  }
}

// One warp per query: k best over the slices.
template <int KPL>
__global__ void k_exact_merge(int64_t nq, int k, int slices, const double* __restrict__ part_dist,
                              const uint32_t* __restrict__ part_idx, double* __restrict__ out_dist,
                              int32_t* __restrict__ out_idx) {
  const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (q >= nq) return;
  const double kInf = __longlong_as_double(0x7FF0000000000000LL);
  WarpList<KPL, double> L;
#pragma unroll
  for (int r = 0; r < KPL; ++r) {
    L.key[r] = kInf;
    L.id[r] = kNoId;
  }
  for (int s = 0; s < slices; ++s) {
    const size_t row = ((size_t)s * nq + q) * k;
    for (int e0 = 0; e0 < k; e0 += 32) {
      const int e = e0 + lane;
      const double ck = e < k ? part_dist[row + e] : kInf;
      const uint32_t ci = e < k ? part_idx[row + e] : kNoId;
      const bool pass = ck < kInf;
      if (__any_sync(0xFFFFFFFFu, pass)) warp_list_insert(L, pass ? ck : kInf, pass ? ci : kNoId);
    }
  }
#pragma unroll
  for (int r = 0; r < KPL; ++r) {
    const int e = r * 32 + lane;
    if (e < k) {
      out_dist[q * k + e] = L.key[r];
      out_idx[q * k + e] = (int32_t)L.id[r];
    }
  }
}

// A slice starts with open lists, whose pairs all get FP64 keys: the filter pays where
// the slice is long against that and k (1088 queries x 25,787 x 14, k=28, slices of
// 759: 2.32 -> 2.11 ms).  Past k = 32 the lists' registers leave one block per SM
// (1721 x 28,652 x 169, k=33, slices of 1365: 7.44 -> 7.03 ms, and slower below).
bool exact_filter_applies(int64_t slice, int k, int d) {
  return slice >= 512 + (k <= 32 ? 8 : 32) * (int64_t)k && d <= kFilterMaxDim;
}

int exact_fp64(const float* X, int64_t n, int d, int dpad, int k, int metric,
               const int64_t* queries, int64_t nq, double* norms, double* part_dist,
               uint32_t* part_idx, int slices, double* out_dist, int32_t* out_idx,
               cudaStream_t st) {
  if (metric == KNN_METRIC_COSINE)
    k_exact_norms<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(X, n, d, dpad, norms);
  const int64_t slice = (n + slices - 1) / slices;
  dim3 grid((unsigned)((nq + kET - 1) / kET), (unsigned)slices);
  const int kpl = kpl_for(k);
  const bool filter = exact_filter_applies(slice, k, d);
  const bool vec = (dpad & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
#define KNN_EXACT(M, KP)                                                                                            \
  do {                                                                                                              \
    /* also where the filter stays off: with lazy loading a kernel's first use may allocate, and one small call  */ \
    /* ahead of time is what lets knn_exact_fp64_noalloc's later ones run in a process without free memory        */ \
    cudaFuncSetAttribute(k_exact_filtered<M, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FilterSmem)); \
    if (filter) {                                                                                                   \
      k_exact_filtered<M, KP><<<grid, 256, sizeof(FilterSmem), st>>>(X, n, d, dpad, vec, k, queries, nq, norms, slice, \
                                                                     part_dist, part_idx);                          \
    }                                                                                                               \
    k_exact<M, KP><<<grid, 256, 0, st>>>(X, n, d, dpad, k, queries, nq, norms, slice, part_dist, part_idx, filter);  \
  } while (0)
#define KNN_EXACT_M(M) \
  do { if (kpl == 1) KNN_EXACT(M, 1); else if (kpl == 2) KNN_EXACT(M, 2); else KNN_EXACT(M, 4); } while (0)
  if (metric == KNN_METRIC_EUCLIDEAN) KNN_EXACT_M(KNN_METRIC_EUCLIDEAN);
  else if (metric == KNN_METRIC_TAXICAB) KNN_EXACT_M(KNN_METRIC_TAXICAB);
  else KNN_EXACT_M(KNN_METRIC_COSINE);
#undef KNN_EXACT_M
#undef KNN_EXACT
  const unsigned mb = (unsigned)((nq * 32 + 255) / 256);
  if (kpl == 1) k_exact_merge<1><<<mb, 256, 0, st>>>(nq, k, slices, part_dist, part_idx, out_dist, out_idx);
  else if (kpl == 2) k_exact_merge<2><<<mb, 256, 0, st>>>(nq, k, slices, part_dist, part_idx, out_dist, out_idx);
  else k_exact_merge<4><<<mb, 256, 0, st>>>(nq, k, slices, part_dist, part_idx, out_dist, out_idx);
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

}  // namespace knn
