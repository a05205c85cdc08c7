// Learned split directions.  A small MLP
//
//   f(x) = W2 gelu(W1 s(x) + b1) + b2,   d -> 256 -> 64,
//   s(x) = (u(x) - mean) * inv_std        (per-dimension, from the sample;
//                                          u(x) = x/|x| for COSINE, else x),
//   gelu(a) = 0.5 a (1 + tanh(sqrt(2/pi) (a + 0.044715 a^3)))
//
// is trained on the GPU with a triplet (contrastive) loss on the k-NN graph
// that the plain method builds for a sample of the points:
//
//   loss = mean_b max(0, margin + |f(a) - f(p)|^2 - |f(a) - f(n)|^2)
//
// (a: a sample point; p: one of its graph neighbours of rank < gk/2; n: either
// a random sample point or a graph neighbour of rank >= gk/2), with Adam.  The
// trees are then built on the 64-dim embeddings f(x), so every split
// direction f(x_p2) - f(x_p1) lives in the learned space; leaf blocks and
// propagation still rank the original rows with exact keys.  The reference has
// no counterpart: its split directions use raw coordinates
// (euclideandistancematrixgpu.cu:2138-2164), which stays the default here.
//
// Everything is FP32 on CUDA cores, every sum in a fixed order, so training is
// deterministic.  A training step is three launches: k_step_rows takes the triplets
// through the network and back, a block per 8 of them; k_step_weight_grads reduces the
// weight gradients over the rows (split-K partials); k_step_finish sums the partials
// and applies Adam.
#include <cmath>
#include <cstring>

#include "knn_internal.cuh"
#include "knn_kernels.cuh"

namespace knn {

namespace {
constexpr int kGT = 64;    // GEMM tile (rows and columns)
constexpr int kGK = 16;    // GEMM k-chunk
constexpr int kSplitK = 8; // row splits of the weight gradients
constexpr int kColSplits = 16;         // and of the bias gradients
constexpr int kTB = 8;                 // triplets per block of k_step_rows,
constexpr int kTR = 3 * kTB;           // their rows: anchors, positives, negatives
constexpr int kHalfR = kTR / 2;        // rows per thread
constexpr int kDChunk = 32;            // dims of the first layer staged at a time
constexpr int kWPitch = kMlpHidden + 1;  // odd: lanes along either index of a weight tile hit different banks
constexpr int kGPitch = kTR + 4;
constexpr float kSqrt2OverPi = 0.7978845608028654f;
constexpr float kGeluC = 0.044715f;
constexpr float kB1 = 0.9f, kB2 = 0.999f, kEps = 1e-8f;
}  // namespace

__device__ __forceinline__ float gelu_f(float a) {
  const float u = kSqrt2OverPi * (a + kGeluC * a * a * a);
  return 0.5f * a * (1.0f + tanhf(u));
}
__device__ __forceinline__ float gelu_grad(float a) {
  const float u = kSqrt2OverPi * (a + kGeluC * a * a * a);
  const float t = tanhf(u);
  const float du = kSqrt2OverPi * (1.0f + 3.0f * kGeluC * a * a);
  return 0.5f * (1.0f + t) + 0.5f * a * (1.0f - t * t) * du;
}

// C[i][j] = sum_k A(i,k) B(j,k) (+ bias[j]) (GELU), with A(i,k) = A[i*sai + k*sak]
// and B(j,k) = B[j*sbj + k*sbk] (the embedding of all points).
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, const float* __restrict__ A, int64_t sai,
                                              int64_t sak, const float* __restrict__ B, int64_t sbj,
                                              int64_t sbk, const float* __restrict__ bias, float* __restrict__ C,
                                              int64_t ldc, int gelu) {
  __shared__ __align__(16) float As[kGK][kGT + 4];
  __shared__ __align__(16) float Bs[kGK][kGT + 4];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int i0 = blockIdx.y * kGT, j0 = blockIdx.x * kGT;
  // Loads walk whichever index is unit-stride.
  const bool a_k_fast = sak <= sai, b_k_fast = sbk <= sbj;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += kGK) {
    for (int e = tid; e < kGT * kGK; e += 256) {
      int r, kk;
      if (a_k_fast) { r = e / kGK; kk = e % kGK; } else { r = e % kGT; kk = e / kGT; }
      const int gi = i0 + r, gk = k0 + kk;
      As[kk][r] = (gi < M && gk < K) ? A[(int64_t)gi * sai + (int64_t)gk * sak] : 0.f;
      if (b_k_fast) { r = e / kGK; kk = e % kGK; } else { r = e % kGT; kk = e / kGT; }
      const int gj = j0 + r, gk2 = k0 + kk;
      Bs[kk][r] = (gj < N && gk2 < K) ? B[(int64_t)gj * sbj + (int64_t)gk2 * sbk] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGK; ++kk) {
      const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = __fmaf_rn(av[p], bv[q], acc[p][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + ty * 4 + p, j = j0 + tx * 4 + q;
      if (i >= M || j >= N) continue;
      float v = acc[p][q];
      if (bias) v = __fadd_rn(v, bias[j]);
      if (gelu) v = gelu_f(v);
      C[(int64_t)i * ldc + j] = v;
    }
}

// Row scale of the network input: 1/|x| for COSINE (norms given; a zero row
// stays zero), else 1.
__device__ __forceinline__ float unit_scale(const float* __restrict__ norms, int64_t i) {
  if (!norms) return 1.0f;
  const float nr = norms[i];
  return nr > 0.f ? __fdiv_rn(1.0f, nr) : 1.0f;
}

// Sample row of triplet b's anchor (role 0: a random sample point), positive (1: a
// graph neighbour of a of rank < half) or negative (2: a random sample point (even
// hash) or a graph neighbour of a of rank >= half (odd hash)).
__device__ __forceinline__ int64_t triplet_source(int64_t ns, const int32_t* __restrict__ graph, int gk, int half,
                                                  uint64_t seed, int step, int b, int role) {
  const uint64_t h = splitmix64(seed ^ splitmix64((uint64_t)step * 0x9E3779B97F4A7C15ull + (uint64_t)b));
  const int64_t a = (int64_t)(h % (uint64_t)ns);
  if (role == 1) {
    const uint64_t h2 = splitmix64(h ^ 0x5851F42D4C957F2Dull);
    return graph[a * gk + (int64_t)(h2 % (uint64_t)half)];
  }
  if (role == 2) {
    const uint64_t h3 = splitmix64(h ^ 0x14057B7EF767814Full);
    if ((h3 & 1) == 0 || gk <= half) return (int64_t)((h3 >> 1) % (uint64_t)ns);
    return graph[a * gk + half + (int64_t)((h3 >> 1) % (uint64_t)(gk - half))];
  }
  return a;
}

// Where a step draws its triplets from (Xs null: the rows are given).
struct TripletSource {
  const float *Xs, *norms, *mean, *inv_std;
  const int32_t* graph;
  int64_t ns;
  int dpad, gk, half;
  uint64_t seed;
};

// What a step hands from kernel to kernel: G1 = gelu(A1) and dA1 [R][H], dZ [R][E]
// (R = 3B: anchors, positives, negatives), hinge[b] = the triplets' losses, and
// the partial sums of dW1, dW2, db1 and db2.
struct StepWs {
  float *G1, *dA, *dZ, *part1, *part2, *cpart1, *cpart2, *hinge;
};

__device__ __forceinline__ void cp_async_f(float* dst, const float* src, bool on) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(src), "r"(on ? 4 : 0) : "memory");
}

struct RowsSmem {
  float w2[kMlpEmbed * kWPitch];         // [e][h]
  float w1[2][kDChunk * kWPitch];        // [c][h]
  float x[2][kDChunk * kTR];             // [c][row]
  float g1[kMlpHidden * kGPitch];        // [h][row]
  float z[kTR * (kMlpEmbed + 1)];        // [row][e]
  float dz[kMlpEmbed * kTR + 8];         // [e][row]
};

// One block takes 8 triplets (24 rows) through f, the loss
//   mean_b max(0, margin + |f(a) - f(p)|^2 - |f(a) - f(n)|^2)
// and back to dA1 = (dZ W2) * gelu'(A1).  All of this is per row, so nothing but
// the weights is read from memory and the step's five launches of the three
// products, the loss and the GELU gradient are one; 1024 triplets are 128
// blocks on 148 SMs.  A thread holds 12 rows x 2 hidden units (one warp-wide
// read of two weights and three broadcast reads per 24 FMAs) and keeps its
// pre-activations in registers until the way back.
//
// What bounds it: shared memory and FMA issue about evenly, at 8 warps per SM.
// 1024 triplets, d = 64, B200: a step 193 us as seventeen launches (the five products
// 31 us each), now 41: this kernel 22.8, k_step_weight_grads 14.0, k_step_finish 4.1.
__global__ void __launch_bounds__(256, 1)
    k_step_rows(TripletSource src, float* __restrict__ rows, int d, int B, float margin, const int* __restrict__ step,
                const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
                const float* __restrict__ b2, StepWs ws) {
  constexpr int H = kMlpHidden, E = kMlpEmbed;
  extern __shared__ __align__(16) unsigned char step_smem[];
  RowsSmem& sm = *reinterpret_cast<RowsSmem*>(step_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b0 = blockIdx.x * kTB;
  for (int i = tid; i < E * H; i += 256) cp_async_f(&sm.w2[(i >> 8) * kWPitch + (i & 255)], W2 + i, true);
  if (src.Xs) {
    const int b = b0 + warp;  // a warp draws one triplet
    if (b < B)
      for (int role = 0; role < 3; ++role) {
        const int64_t i = triplet_source(src.ns, src.graph, src.gk, src.half, src.seed, *step, b, role);
        const float sc = unit_scale(src.norms, i);
        float* out = rows + ((int64_t)role * B + b) * d;
        for (int c = lane; c < d; c += 32)
          out[c] = __fmul_rn(__fsub_rn(__fmul_rn(src.Xs[i * src.dpad + c], sc), src.mean[c]), src.inv_std[c]);
      }
    __syncthreads();  // the rows are read back by the whole block
  }
  auto stage = [&](int ch, int buf) {
    for (int i = tid; i < kDChunk * H; i += 256) {
      const int c = i & 31, h = i >> 5, dim = ch * kDChunk + c;
      cp_async_f(&sm.w1[buf][c * kWPitch + h], W1 + (dim < d ? (int64_t)h * d + dim : 0), dim < d);
    }
    for (int i = tid; i < kDChunk * kTR; i += 256) {
      const int c = i & 31, l = i >> 5, dim = ch * kDChunk + c, b = b0 + (l & (kTB - 1));
      const bool on = dim < d && b < B;
      cp_async_f(&sm.x[buf][c * kTR + l], rows + (on ? ((int64_t)(l / kTB) * B + b) * d + dim : 0), on);
    }
    cp_async_commit();
  };
  // A1 = rows W1^T + b1, hidden units tx and tx + 128 of rows 12 rg .. 12 rg + 11
  const int tx = tid & 127, rg = tid >> 7;
  float pre[kHalfR][2] = {};
  auto outer = [&](const float* a, float w0, float w1) {
    const float4* a4 = reinterpret_cast<const float4*>(a);
#pragma unroll
    for (int u = 0; u < kHalfR / 4; ++u) {
      const float4 v = a4[u];
      const float av[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        pre[4 * u + i][0] = __fmaf_rn(av[i], w0, pre[4 * u + i][0]);
        pre[4 * u + i][1] = __fmaf_rn(av[i], w1, pre[4 * u + i][1]);
      }
    }
  };
  const int nch = (d + kDChunk - 1) / kDChunk;
  stage(0, 0);
  for (int ch = 0; ch < nch; ++ch) {
    const int buf = ch & 1;
    if (ch + 1 < nch) {
      stage(ch + 1, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll 8
    for (int c = 0; c < kDChunk; ++c)
      outer(&sm.x[buf][c * kTR + rg * kHalfR], sm.w1[buf][c * kWPitch + tx], sm.w1[buf][c * kWPitch + tx + 128]);
    __syncthreads();  // the buffer is refilled by the next round
  }
  auto row_of = [&](int l) { return (int64_t)(l / kTB) * B + b0 + (l & (kTB - 1)); };
  auto on = [&](int l) { return b0 + (l & (kTB - 1)) < B; };
  {
    const float c0 = b1[tx], c1 = b1[tx + 128];
#pragma unroll
    for (int i = 0; i < kHalfR; ++i) {
      const int l = rg * kHalfR + i;
      pre[i][0] = __fadd_rn(pre[i][0], c0);
      pre[i][1] = __fadd_rn(pre[i][1], c1);
      const float g0 = gelu_f(pre[i][0]), g1 = gelu_f(pre[i][1]);
      sm.g1[tx * kGPitch + l] = g0;
      sm.g1[(tx + 128) * kGPitch + l] = g1;
      if (on(l)) {
        ws.G1[row_of(l) * H + tx] = g0;
        ws.G1[row_of(l) * H + tx + 128] = g1;
      }
    }
  }
  __syncthreads();
  // Z = G1 W2^T + b2: output tid & 63 of 12 rows; four warps, as 6 rows each of
  // eight would double the shared-memory reads that bound this part
  if (tid < 128) {
    const int e = tid & 63, r0 = (tid >> 6) * kHalfR;
    float acc[kHalfR] = {};
#pragma unroll 8
    for (int h = 0; h < H; ++h) {
      const float w = sm.w2[e * kWPitch + h];
      const float4* a4 = reinterpret_cast<const float4*>(&sm.g1[h * kGPitch + r0]);
#pragma unroll
      for (int u = 0; u < kHalfR / 4; ++u) {
        const float4 v = a4[u];
        acc[4 * u] = __fmaf_rn(v.x, w, acc[4 * u]);
        acc[4 * u + 1] = __fmaf_rn(v.y, w, acc[4 * u + 1]);
        acc[4 * u + 2] = __fmaf_rn(v.z, w, acc[4 * u + 2]);
        acc[4 * u + 3] = __fmaf_rn(v.w, w, acc[4 * u + 3]);
      }
    }
    const float bias = b2[e];
#pragma unroll
    for (int i = 0; i < kHalfR; ++i) sm.z[(r0 + i) * (E + 1) + e] = __fadd_rn(acc[i], bias);
  }
  __syncthreads();
  // the loss and dZ, a warp per triplet
  {
    const int b = b0 + warp;
    const float* za = sm.z + warp * (E + 1);
    const float* zp = za + kTB * (E + 1);
    const float* zn = zp + kTB * (E + 1);
    float dap = 0.f, dan = 0.f;
    for (int e = lane; e < E; e += 32) {
      const float u = za[e] - zp[e], w = za[e] - zn[e];
      dap = __fmaf_rn(u, u, dap);
      dan = __fmaf_rn(w, w, dan);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      dap += __shfl_xor_sync(0xFFFFFFFFu, dap, off);
      dan += __shfl_xor_sync(0xFFFFFFFFu, dan, off);
    }
    const float l = margin + dap - dan;
    const float s = l > 0.f ? 2.0f / (float)B : 0.f;
    // d/dza = 2(za-zp) - 2(za-zn), d/dzp = -2(za-zp), d/dzn = 2(za-zn)
    for (int e = lane; e < E; e += 32) {
      const float u = za[e] - zp[e], w = za[e] - zn[e];
      const float ga = s * (u - w), gp = -s * u, gn = s * w;
      sm.dz[e * kTR + warp] = ga;
      sm.dz[e * kTR + kTB + warp] = gp;
      sm.dz[e * kTR + 2 * kTB + warp] = gn;
      if (b < B) {
        ws.dZ[(int64_t)b * E + e] = ga;
        ws.dZ[(int64_t)(B + b) * E + e] = gp;
        ws.dZ[(int64_t)(2 * B + b) * E + e] = gn;
      }
    }
    if (lane == 0 && b < B) ws.hinge[b] = l > 0.f ? l : 0.f;
  }
  __syncthreads();
  // dA1 = (dZ W2) * gelu'(A1)
  float grad[kHalfR][2];
#pragma unroll
  for (int i = 0; i < kHalfR; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      grad[i][j] = gelu_grad(pre[i][j]);
      pre[i][j] = 0.f;
    }
#pragma unroll 8
  for (int e = 0; e < E; ++e)
    outer(&sm.dz[e * kTR + rg * kHalfR], sm.w2[e * kWPitch + tx], sm.w2[e * kWPitch + tx + 128]);
#pragma unroll
  for (int i = 0; i < kHalfR; ++i) {
    const int l = rg * kHalfR + i;
    if (!on(l)) continue;
    ws.dA[row_of(l) * H + tx] = __fmul_rn(pre[i][0], grad[i][0]);
    ws.dA[row_of(l) * H + tx + 128] = __fmul_rn(pre[i][1], grad[i][1]);
  }
}

// Partial sums over the rows, a block of 128 threads per job:
//   dW2[e][h] = sum_r dZ[r][e] G1[r][h], dW1[h][c] = sum_r dA1[r][h] rows[r][c]:
//     tiles of 32 x 64 outputs x one of kSplitK row ranges, 4 x 4 outputs a thread;
//   db1, db2: 32 columns x one of kColSplits row ranges, 8 row lanes per column
//     combined in a fixed order.
// One launch for all: 288 blocks at d = 64, where the two products alone were 32
// blocks of 64 x 64 each.  Advances the step counter, which no block here reads.
constexpr int kWM = 32, kWN = 64, kWR = 32;  // weight-gradient tile and rows per stage
__global__ void __launch_bounds__(128) k_step_weight_grads(const float* __restrict__ rows, int d, int R, StepWs ws,
                                                           int* __restrict__ step) {
  constexpr int H = kMlpHidden, E = kMlpEmbed;
  __shared__ __align__(16) float As[2][kWR][kWM];
  __shared__ __align__(16) float Bs[2][kWR][kWN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0 && tid == 0 && step) *step += 1;
  constexpr int jobs2 = (E / kWM) * (H / kWN) * kSplitK;
  const int nt = (d + kWN - 1) / kWN, jobs1 = (H / kWM) * nt * kSplitK;
  int job = blockIdx.x;
  if (job >= jobs2 + jobs1) {
    job -= jobs2 + jobs1;
    const int z = job / ((H + E) / 32), x = job % ((H + E) / 32);
    const bool first = x < H / 32;
    const float* G = first ? ws.dA : ws.dZ;
    const int N = first ? H : E, j = (first ? x : x - H / 32) * 32 + lane;
    const int per = (R + kColSplits - 1) / kColSplits;
    const int r0 = z * per, r1 = min(R, r0 + per);
    float(*red)[kWM] = As[0];
    for (int y = warp; y < 8; y += 4) {
      float s = 0.f;
      for (int i = r0 + y; i < r1; i += 8) s = __fadd_rn(s, G[(int64_t)i * N + j]);
      red[y][lane] = s;
    }
    __syncthreads();
    if (warp == 0) {
      float t = red[0][lane];
      for (int q = 1; q < 8; ++q) t = __fadd_rn(t, red[q][lane]);
      (first ? ws.cpart1 : ws.cpart2)[(int64_t)z * N + j] = t;
    }
    return;
  }
  const bool second = job < jobs2;
  if (!second) job -= jobs2;
  const float* A = second ? ws.dZ : ws.dA;
  const float* Bm = second ? ws.G1 : rows;
  const int M = second ? E : H, N = second ? H : d, cols = second ? H / kWN : nt;
  const int z = job % kSplitK, tile = job / kSplitK, m0 = (tile / cols) * kWM, n0 = (tile % cols) * kWN;
  const int per = (((R + kSplitK - 1) / kSplitK) + kGK - 1) / kGK * kGK;
  const int kb = z * per, ke = min(R, kb + per);
  const bool quads = (N & 3) == 0;  // 16-byte rows
  auto stage = [&](int k0, int buf) {
    for (int i = tid; i < kWR * kWM / 4; i += 128) {
      const int r = i / (kWM / 4), c = (i % (kWM / 4)) * 4;
      cp_async16(&As[buf][r][c], A + (k0 + r < ke ? (int64_t)(k0 + r) * M + m0 + c : 0), k0 + r < ke ? 16 : 0);
    }
    if (quads) {
      for (int i = tid; i < kWR * kWN / 4; i += 128) {
        const int r = i / (kWN / 4), c = (i % (kWN / 4)) * 4;
        const bool on = k0 + r < ke && n0 + c < N;
        cp_async16(&Bs[buf][r][c], Bm + (on ? (int64_t)(k0 + r) * N + n0 + c : 0), on ? 16 : 0);
      }
    } else {
      for (int i = tid; i < kWR * kWN; i += 128) {
        const int r = i / kWN, c = i % kWN;
        const bool on = k0 + r < ke && n0 + c < N;
        cp_async_f(&Bs[buf][r][c], Bm + (on ? (int64_t)(k0 + r) * N + n0 + c : 0), on);
      }
    }
    cp_async_commit();
  };
  const int tx = lane & 15, ty = warp * 2 + (lane >> 4);
  float acc[4][4] = {};
  if (kb < ke) stage(kb, 0);
  int buf = 0;
  for (int k0 = kb; k0 < ke; k0 += kWR, buf ^= 1) {
    if (k0 + kWR < ke) {
      stage(k0 + kWR, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < kWR; ++r) {
      const float4 a = *reinterpret_cast<const float4*>(&As[buf][r][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[buf][r][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = __fmaf_rn(av[p], bv[q], acc[p][q]);
    }
    __syncthreads();
  }
  float* C = (second ? ws.part2 : ws.part1) + (int64_t)z * M * N;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (n0 + tx * 4 + q < N) C[(int64_t)(m0 + ty * 4 + p) * N + n0 + tx * 4 + q] = acc[p][q];
}

// Gradients = the partial sums added in order, for Adam on the parameters w (m, v;
// *step = the step's number, from 1) or, without w, to `out`.  The last block writes
// the step's mean loss, the hinges summed in a fixed order.
__global__ void __launch_bounds__(256) k_step_finish(StepWs ws, int d, int B, float* __restrict__ out,
                                                     float* __restrict__ w, float* __restrict__ m,
                                                     float* __restrict__ v, float lr, const int* __restrict__ step,
                                                     float* __restrict__ loss) {
  constexpr int H = kMlpHidden, E = kMlpEmbed;
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ float red[256];
    float s = 0.f;
    for (int b = threadIdx.x; b < B; b += 256) s = __fadd_rn(s, ws.hinge[b]);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int u = 128; u >= 1; u >>= 1) {
      if ((int)threadIdx.x < u) red[threadIdx.x] = __fadd_rn(red[threadIdx.x], red[threadIdx.x + u]);
      __syncthreads();
    }
    if (threadIdx.x == 0) loss[step ? *step - 1 : 0] = red[0] / (float)B;
    return;
  }
  // parameters: W1 [H][d], b1 [H], W2 [E][H], b2 [E]
  const int64_t n1 = (int64_t)H * d, n2 = (int64_t)E * H;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float* part;
  int64_t at = i, count;
  int splits = kSplitK;
  if (at < n1) {
    part = ws.part1;
    count = n1;
  } else if ((at -= n1) < H) {
    part = ws.cpart1;
    count = H;
    splits = kColSplits;
  } else if ((at -= H) < n2) {
    part = ws.part2;
    count = n2;
  } else if ((at -= n2) < E) {
    part = ws.cpart2;
    count = E;
    splits = kColSplits;
  } else {
    return;
  }
  float gi = part[at];
#pragma unroll 8
  for (int z = 1; z < splits; ++z) gi = __fadd_rn(gi, part[(int64_t)z * count + at]);
  if (!w) {
    out[i] = gi;
    return;
  }
  const float t = (float)(*step);
  const float c1 = 1.0f - powf(kB1, t), c2 = 1.0f - powf(kB2, t);
  const float mi = kB1 * m[i] + (1.f - kB1) * gi;
  const float vi = kB2 * v[i] + (1.f - kB2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + kEps);
}

// Per-dimension mean and 1/std of the sample rows, one warp and block per
// dimension.  A lane's sums are serial chains; the rows of sixteen steps are read
// ahead of them (65,536 rows x 64 on a B200: 567 us reading one at a time,
// 228 us now).
__global__ void __launch_bounds__(32) k_standardise_stats(const float* __restrict__ Xs,
                                                          const float* __restrict__ norms, int dpad, int d,
                                                          int64_t ns, float* __restrict__ mean,
                                                          float* __restrict__ inv_std) {
  constexpr int kAhead = 16;
  const int c = blockIdx.x, lane = threadIdx.x;
  double s = 0, s2 = 0;
  for (int64_t i0 = lane; i0 < ns; i0 += 32 * kAhead) {
    float x[kAhead], nr[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t i = i0 + 32 * u;
      x[u] = i < ns ? __ldg(Xs + i * dpad + c) : 0.f;
      nr[u] = norms && i < ns ? __ldg(norms + i) : 1.f;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (i0 + 32 * u >= ns) break;
      const double v = __fmul_rn(x[u], nr[u] > 0.f ? __fdiv_rn(1.0f, nr[u]) : 1.0f);
      s += v;
      s2 += v * v;
    }
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    s += __shfl_xor_sync(0xFFFFFFFFu, s, off);
    s2 += __shfl_xor_sync(0xFFFFFFFFu, s2, off);
  }
  if (lane == 0) {
    const double mu = s / (double)ns;
    const double var = s2 / (double)ns - mu * mu;
    mean[c] = (float)mu;
    inv_std[c] = var > 1e-12 ? (float)(1.0 / sqrt(var)) : 1.0f;
  }
}

// Rows [r0, r0+m) of X, standardised, into a dense [m][d] block.
__global__ void k_standardise_rows(const float* __restrict__ X, const float* __restrict__ norms, int dpad, int d,
                                   int64_t r0, int m, const float* __restrict__ mean,
                                   const float* __restrict__ inv_std, float* __restrict__ out) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (int64_t)m * d) return;
  const int64_t r = g / d;
  const int c = (int)(g - r * d);
  const float sc = unit_scale(norms, r0 + r);
  out[g] = __fmul_rn(__fsub_rn(__fmul_rn(X[(size_t)(r0 + r) * dpad + c], sc), mean[c]), inv_std[c]);
}

// Gaussian initial weights (Box-Muller on a splitmix64 stream) times `scale`.
__global__ void k_init_normal(float* __restrict__ w, int64_t count, float scale, uint64_t seed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint64_t h = splitmix64(seed + (uint64_t)i * 0x9E3779B97F4A7C15ull);
  const float u1 = ((float)((h >> 40) & 0xFFFFFF) + 1.0f) / 16777217.0f;
  const float u2 = (float)((h >> 16) & 0xFFFFFF) / 16777216.0f;
  w[i] = scale * sqrtf(-2.0f * logf(u1)) * cosf(6.283185307179586f * u2);
}

// Sample rows: row i of Xs = row floor(i * n / ns) of X (padded rows).
__global__ void k_gather_sample(const float* __restrict__ X, int64_t n, int dpad, int64_t ns,
                                float* __restrict__ Xs) {
  const int q = dpad / 4;
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ns * q) return;
  const int64_t i = g / q;
  const int c4 = (int)(g - i * q);
  const int64_t src = (int64_t)(((unsigned __int128)i * (unsigned __int128)n) / (unsigned __int128)ns);
  reinterpret_cast<float4*>(Xs)[g] = reinterpret_cast<const float4*>(X + src * dpad)[c4];
}

namespace {

inline unsigned blocks_for(int64_t count, int threads) { return (unsigned)((count + threads - 1) / threads); }

void gemm(cudaStream_t st, int M, int N, int K, const float* A, int64_t sai, int64_t sak, const float* B,
          int64_t sbj, int64_t sbk, const float* bias, float* C, int64_t ldc, int gelu) {
  dim3 grid((N + kGT - 1) / kGT, (M + kGT - 1) / kGT, 1);
  k_gemm<<<grid, 256, 0, st>>>(M, N, K, A, sai, sak, B, sbj, sbk, bias, C, ldc, gelu);
}

struct MlpParams {
  float* W1;
  float* b1;
  float* W2;
  float* b2;
};

MlpParams param_view(float* p, int d) {
  MlpParams q;
  q.W1 = p;
  q.b1 = q.W1 + (size_t)kMlpHidden * d;
  q.W2 = q.b1 + kMlpHidden;
  q.b2 = q.W2 + (size_t)kMlpEmbed * kMlpHidden;
  return q;
}

// Every part a multiple of 4 floats but the hinges, which come last.
StepWs ws_view(float* ws, int d, int R) {
  StepWs w;
  w.G1 = ws;
  w.dA = w.G1 + (size_t)R * kMlpHidden;
  w.dZ = w.dA + (size_t)R * kMlpHidden;
  w.part1 = w.dZ + (size_t)R * kMlpEmbed;
  w.part2 = w.part1 + (size_t)kSplitK * kMlpHidden * d;
  w.cpart1 = w.part2 + (size_t)kSplitK * kMlpEmbed * kMlpHidden;
  w.cpart2 = w.cpart1 + (size_t)kColSplits * kMlpHidden;
  w.hinge = w.cpart2 + (size_t)kColSplits * kMlpEmbed;
  return w;
}

// One forward + backward over the rows (drawn from `src`, or given), then Adam on
// the parameters (adam_m set) or the gradient to `grad`.
void run_step(cudaStream_t st, float* params, int d, const TripletSource& src, float* rows, int B, float margin,
              float* grad, float* adam_m, float* adam_v, float lr, float* ws, int* step, float* loss,
              LaunchLog& log) {
  const MlpParams p = param_view(params, d);
  const StepWs w = ws_view(ws, d, 3 * B);
  cudaFuncSetAttribute(k_step_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RowsSmem));
  k_step_rows<<<blocks_for(B, kTB), 256, sizeof(RowsSmem), st>>>(src, rows, d, B, margin, step, p.W1, p.b1, p.W2, p.b2,
                                                                 w);
  const int jobs = (kMlpEmbed / kWM) * (kMlpHidden / kWN) * kSplitK +
                   (kMlpHidden / kWM) * ((d + kWN - 1) / kWN) * kSplitK +
                   (kMlpHidden + kMlpEmbed) / 32 * kColSplits;
  k_step_weight_grads<<<jobs, 128, 0, st>>>(rows, d, 3 * B, w, step);
  const int64_t np = (int64_t)mlp_param_count(d);
  k_step_finish<<<blocks_for(np, 256) + 1, 256, 0, st>>>(w, d, B, grad, adam_m ? params : nullptr, adam_m, adam_v, lr,
                                                         step, loss);
  log.add(3);
}

}  // namespace

size_t mlp_param_count(int d) {
  return (size_t)kMlpHidden * d + kMlpHidden + (size_t)kMlpEmbed * kMlpHidden + kMlpEmbed;
}

size_t mlp_fwd_bwd_ws_floats(int d, int B) {
  const size_t R = 3 * (size_t)B;
  const size_t all = R * (2 * kMlpHidden + kMlpEmbed) + (size_t)kSplitK * kMlpHidden * ((size_t)d + kMlpEmbed) +
                     (size_t)kColSplits * (kMlpHidden + kMlpEmbed) + (size_t)B;
  return (all + 3) & ~(size_t)3;
}

size_t mlp_train_ws_floats(int d, int B) {
  return mlp_fwd_bwd_ws_floats(d, B) + (size_t)3 * B * d + 2 * mlp_param_count(d) + 64;
}

int mlp_train(const MlpTrainArgs& a, LaunchLog& log) {
  cudaStream_t st = a.stream;
  const size_t np = mlp_param_count(a.d);
  const int B = a.batch;
  float* fb = a.ws;
  float* rows = fb + mlp_fwd_bwd_ws_floats(a.d, B);
  float* adam_m = rows + (size_t)3 * B * a.d;
  float* adam_v = adam_m + np;
  int* step = reinterpret_cast<int*>(adam_v + np);

  const MlpParams p = param_view(a.params, a.d);
  k_init_normal<<<blocks_for((int64_t)kMlpHidden * a.d, 256), 256, 0, st>>>(
      p.W1, (int64_t)kMlpHidden * a.d, 1.0f / sqrtf((float)a.d), a.seed);
  k_init_normal<<<blocks_for((int64_t)kMlpEmbed * kMlpHidden, 256), 256, 0, st>>>(
      p.W2, (int64_t)kMlpEmbed * kMlpHidden, 1.0f / sqrtf((float)kMlpHidden), a.seed ^ 0xA5A5A5A5ull);
  if (cudaMemsetAsync(p.b1, 0, sizeof(float) * kMlpHidden, st) != cudaSuccess ||
      cudaMemsetAsync(p.b2, 0, sizeof(float) * kMlpEmbed, st) != cudaSuccess ||
      cudaMemsetAsync(adam_m, 0, sizeof(float) * 2 * np + sizeof(int), st) != cudaSuccess ||
      cudaMemsetAsync(a.loss, 0, sizeof(float) * (size_t)(a.steps > 0 ? a.steps : 1), st) != cudaSuccess)
    return KNN_ERR_CUDA;
  k_standardise_stats<<<a.d, 32, 0, st>>>(a.Xs, a.norms, a.dpad, a.d, a.ns, a.mean, a.inv_std);
  log.add(3);
  const int half = a.gk >= 2 ? a.gk / 2 : 1;
  // The kernels of a step outlast their launches, so plain launches keep the GPU busy
  // and, unlike a captured step, leave no graph to wait for and release.  The step
  // index lives on the device, where k_step_weight_grads advances it.
  const TripletSource src{a.Xs, a.norms, a.mean, a.inv_std, a.graph, a.ns, a.dpad, a.gk, half, a.seed};
  for (int s = 0; s < a.steps; ++s)
    run_step(st, a.params, a.d, src, rows, B, a.margin, nullptr, adam_m, adam_v, a.lr, fb, step, a.loss, log);
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

size_t mlp_embed_ws_floats(int d, int64_t chunk) { return (size_t)chunk * ((size_t)d + kMlpHidden); }

int mlp_embed(const float* X, const float* norms, int64_t n, int d, int dpad, const float* params,
              const float* mean, const float* inv_std, float* ws, int64_t chunk, float* Z, cudaStream_t st,
              LaunchLog& log) {
  const MlpParams p = param_view(const_cast<float*>(params), d);
  float* S = ws;                      // [chunk][d]
  float* G1 = S + (size_t)chunk * d;  // [chunk][H]
  for (int64_t r0 = 0; r0 < n; r0 += chunk) {
    const int m = (int)(n - r0 < chunk ? n - r0 : chunk);
    k_standardise_rows<<<blocks_for((int64_t)m * d, 256), 256, 0, st>>>(X, norms, dpad, d, r0, m, mean, inv_std,
                                                                          S);
    gemm(st, m, kMlpHidden, d, S, d, 1, p.W1, d, 1, p.b1, G1, kMlpHidden, 1);
    gemm(st, m, kMlpEmbed, kMlpHidden, G1, kMlpHidden, 1, p.W2, kMlpHidden, 1, p.b2, Z + (size_t)r0 * kMlpEmbed,
         kMlpEmbed, 0);
    log.add(3);
  }
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

int mlp_loss_grad(const float* params, int d, const float* rows, int B, float margin, float* grad, float* ws,
                  float* loss, cudaStream_t st, LaunchLog& log) {
  // the rows and the parameters are only read: no source to draw from, no Adam
  run_step(st, const_cast<float*>(params), d, TripletSource{}, const_cast<float*>(rows), B, margin, grad, nullptr,
           nullptr, 0.f, ws, nullptr, loss, log);
  return cudaPeekAtLastError() == cudaSuccess ? KNN_OK : KNN_ERR_CUDA;
}

void launch_gather_sample(const float* X, int64_t n, int dpad, int64_t ns, float* Xs, cudaStream_t st) {
  k_gather_sample<<<blocks_for(ns * (dpad / 4), 256), 256, 0, st>>>(X, n, dpad, ns, Xs);
}

}  // namespace knn
