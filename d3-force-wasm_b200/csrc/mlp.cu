// mlp.cu — the learned correction's network (no reference counterpart): a
// per-leaf MLP 12 -> 64 -> 64 -> 2 with GELU, BF16 weights and FP32
// accumulation, and its training (forward, backward and Adam) on the GPU.
//
// Parameters, one float vector (the FP32 master copy; every use rounds the
// weights to bf16, biases stay FP32), weights stored [out][in]:
//   W1 [64][12] | b1 [64] | W2 [64][64] | b2 [64] | W3 [2][64] | b3 [2]
//
// Training (CUDA cores, FP32): a CTA of 256 threads takes tiles of 64 samples;
// the three 64 x 64 x 64 products of a tile (layer 2 forward, its input
// gradient, its weight gradient) and layer 1 are register tiles of 4 x 4 over
// operands in shared memory, both k-major; gelu' and the gradient sums stay
// in registers over all of a CTA's tiles. The CTAs' sums are added in CTA
// order by the kernel that applies them (the result does not depend on
// timing). Loss: mean over samples of sum_o (y_o - t_o)^2.
// Inference (tcgen05, mlp_infer_tc): a CTA per 128 samples, the three layers
// as MMAs of M = 128 with the activations staged as bf16 in shared memory,
// GELU and the biases applied between them from the TMEM accumulators.
#include <cuda_bf16.h>

#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "mlp.cuh"
#include "tc.cuh"

namespace d3 {
namespace {

constexpr int TT = 128;       // samples per inference tile

__device__ __forceinline__ float bf(float w) { return __bfloat162float(__float2bfloat16(w)); }
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678f)); }
__device__ __forceinline__ float gelu_d(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678f)) + z * 0.39894228f * expf(-0.5f * z * z);
}

constexpr int GT = 64;            // samples per training tile
constexpr int GTHREADS = 256;     // 16 x 16 threads, 4 samples x 4 units each
constexpr int PART = (MLP_PARAMS + 1 + 31) / 32 * 32;  // a CTA's sums: the gradient, then the loss
static_assert(MLP_H == GT, "the tiles are square");

// Rows are read 16 bytes at a time; GS floats a row (17 x 16 bytes), so the
// rows that a warp's lanes read or write side by side start in other banks.
constexpr int GS = 68;
struct TrainSmem {
  float w1t[MLP_IN][GS];              // bf16-rounded, [in][out]
  float w2[MLP_H][GS], w2t[MLP_H][GS];  // [out][in] and [in][out]
  float w3[MLP_OUT][GS];
  float a1[GT][GS], a2[GT][GS];       // a row per sample
  float d1[GT][GS], d2[GT][GS];       // dz1, dz2
  float x[GT][MLP_IN];
  float b1[MLP_H], b2[MLP_H];
  float dy[MLP_OUT][GT];
  float b3[MLP_OUT], loss[GTHREADS / 32];
};
static_assert(offsetof(TrainSmem, w2) % 16 == 0 && offsetof(TrainSmem, w2t) % 16 == 0 &&
                  offsetof(TrainSmem, w3) % 16 == 0 && offsetof(TrainSmem, a1) % 16 == 0 &&
                  offsetof(TrainSmem, a2) % 16 == 0 && offsetof(TrainSmem, d1) % 16 == 0 &&
                  offsetof(TrainSmem, d2) % 16 == 0 && offsetof(TrainSmem, x) % 16 == 0 &&
                  MLP_IN % 4 == 0 && GS % 4 == 0,
              "16-byte rows");

// c[i][j] += sum_k A[i0 + i][k] B[k][j0 + j]; A's rows `stride` floats apart.
template <int K>
__device__ __forceinline__ void tile_product(const float *A, int stride, const float (*B)[GS], int i0,
                                             int j0, float c[4][4]) {
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = *reinterpret_cast<const float4 *>(A + (i0 + i) * stride + k);
      a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 b = *reinterpret_cast<const float4 *>(&B[k + q][j0]);
      const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] += a[i][q] * bv[j];
    }
  }
}

// c[i][j] += sum_s A[s][i0 + i] B[s][j0 + j]
__device__ __forceinline__ void tile_outer(const float (*A)[GS], const float (*B)[GS], int i0, int j0,
                                           float c[4][4]) {
#pragma unroll 8
  for (int s = 0; s < GT; ++s) {
    const float4 a = *reinterpret_cast<const float4 *>(&A[s][i0]);
    const float4 b = *reinterpret_cast<const float4 *>(&B[s][j0]);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) c[i][j] += av[i] * bv[j];
  }
}

__device__ __forceinline__ void put_tile(const float v[4][4], int i0, int j0, float (*R)[GS]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4 *>(&R[i0 + i][j0]) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
}

// Sums over samples [0, n) of the per-sample loss and its gradient divided by
// `norm`: each CTA's own into part[blockIdx][PART].
//
// A step of 8,192 samples (128 tiles, an SM each) takes 26 us with its Adam
// kernel (127 us before: 64 CTAs of a thread per sample, atomic gradient
// sums, a host synchronisation per step); it is bound by the tile's chain of
// products (3 x 1,024 FMA a thread) and the 32 erf and exp a thread takes.
__global__ void __launch_bounds__(GTHREADS) k_mlp_grad(const float *x, const float *y, uint32_t n,
                                                       const float *params, float norm, float *part) {
  extern __shared__ __align__(16) float mlp_smem[];
  TrainSmem &S = *reinterpret_cast<TrainSmem *>(mlp_smem);
  const int t = threadIdx.x, i0 = (t >> 4) * 4, j0 = (t & 15) * 4;
  for (int e = t; e < MLP_H * MLP_IN; e += GTHREADS) S.w1t[e % MLP_IN][e / MLP_IN] = bf(params[P_W1 + e]);
  for (int e = t; e < MLP_H * MLP_H; e += GTHREADS) {
    const float w = bf(params[P_W2 + e]);
    S.w2[e / MLP_H][e % MLP_H] = w;
    S.w2t[e % MLP_H][e / MLP_H] = w;
  }
  for (int e = t; e < MLP_OUT * MLP_H; e += GTHREADS) S.w3[e / MLP_H][e % MLP_H] = bf(params[P_W3 + e]);
  if (t < MLP_H) {
    S.b1[t] = params[P_B1 + t];
    S.b2[t] = params[P_B2 + t];
  }
  if (t < MLP_OUT) S.b3[t] = params[P_B3 + t];
  const float inv = 1.f / norm;
  // gradient sums: W2 tile (rows i0.., columns j0..), W1 (row gj, columns gk ..
  // gk + 2), W3 and the biases by the threads that take their columns (gc: a
  // thread's one of W3, b2 and b3). A tile's sum is formed by itself and then
  // added: one chain over all of a CTA's samples would lose bits as it grows
  // (64 tiles of equal terms: 6e-5 of the sum for 2e-6).
  const int gj = t & 63, gk = (t >> 6) * 3;
  float gw2[4][4] = {}, gw1[3] = {}, gb1 = 0, gc = 0, my_loss = 0;
  for (uint32_t base = blockIdx.x * GT; base < n; base += gridDim.x * GT) {
    __syncthreads();  // the weights; the last tile's reads
    for (int e = t; e < GT * MLP_IN; e += GTHREADS) {
      const uint32_t i = base + e / MLP_IN;
      S.x[e / MLP_IN][e % MLP_IN] = i < n ? bf(x[(size_t)base * MLP_IN + e]) : 0.f;
    }
    __syncthreads();
    // layer 1
    float g1[4][4], g2[4][4], v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = S.b1[j0 + j];
    tile_product<MLP_IN>(&S.x[0][0], MLP_IN, S.w1t, i0, j0, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g1[i][j] = gelu_d(v[i][j]);
        v[i][j] = bf(gelu(v[i][j]));
      }
    put_tile(v, i0, j0, S.a1);
    __syncthreads();
    // layer 2
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = S.b2[j0 + j];
    tile_product<MLP_H>(&S.a1[0][0], GS, S.w2t, i0, j0, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g2[i][j] = gelu_d(v[i][j]);
        v[i][j] = bf(gelu(v[i][j]));
      }
    put_tile(v, i0, j0, S.a2);
    __syncthreads();
    // the output layer, a thread per sample and output
    if (t < MLP_OUT * GT) {
      const int smp = t & 63, o = t >> 6;
      const uint32_t i = base + smp;
      float z = S.b3[o];
#pragma unroll 4
      for (int k = 0; k < MLP_H; k += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(&S.a2[smp][k]);
        const float4 w = *reinterpret_cast<const float4 *>(&S.w3[o][k]);
        z += w.x * a.x;
        z += w.y * a.y;
        z += w.z * a.z;
        z += w.w * a.w;
      }
      const float d = i < n ? z - y[(size_t)i * MLP_OUT + o] : 0.f;
      my_loss += d * d;
      S.dy[o][smp] = 2.f * d * inv;
    }
    __syncthreads();
    // dz2 = (W3^T dy) gelu'(z2)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[i][j] = g2[i][j] * fmaf(S.w3[1][j0 + j], S.dy[1][i0 + i], S.w3[0][j0 + j] * S.dy[0][i0 + i]);
    put_tile(v, i0, j0, S.d2);
    __syncthreads();
    // dz1 = (W2^T dz2) gelu'(z1); W2's gradient over the tile's samples
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = 0;
    tile_product<MLP_H>(&S.d2[0][0], GS, S.w2, i0, j0, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] *= g1[i][j];
    put_tile(v, i0, j0, S.d1);
    float tw2[4][4] = {};
    tile_outer(S.d2, S.a1, i0, j0, tw2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) gw2[i][j] += tw2[i][j];
    __syncthreads();
    // the other gradients, a column of samples each
    float tw1[3] = {}, tb1 = 0, tc = 0;
    for (int s = 0; s < GT; ++s) {
      const float d = S.d1[s][gj];
      if (gk == 0) tb1 += d;
#pragma unroll
      for (int q = 0; q < 3; ++q) tw1[q] += d * S.x[s][gk + q];
    }
    gb1 += tb1;
#pragma unroll
    for (int q = 0; q < 3; ++q) gw1[q] += tw1[q];
    if (t < MLP_OUT * MLP_H) {
      const int o = t / MLP_H, k = t % MLP_H;
      for (int s = 0; s < GT; ++s) tc += S.dy[o][s] * S.a2[s][k];
    } else if (t < MLP_OUT * MLP_H + MLP_H) {
      for (int s = 0; s < GT; ++s) tc += S.d2[s][t - MLP_OUT * MLP_H];
    } else if (t < MLP_OUT * MLP_H + MLP_H + MLP_OUT) {
      for (int s = 0; s < GT; ++s) tc += S.dy[t - MLP_OUT * MLP_H - MLP_H][s];
    }
    gc += tc;
  }
  float *g = part + (size_t)blockIdx.x * PART;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) g[P_W2 + (i0 + i) * MLP_H + j0 + j] = gw2[i][j];
#pragma unroll
  for (int q = 0; q < 3; ++q) g[P_W1 + gj * MLP_IN + gk + q] = gw1[q];
  if (gk == 0) g[P_B1 + gj] = gb1;
  if (t < MLP_OUT * MLP_H) g[P_W3 + t] = gc;
  else if (t < MLP_OUT * MLP_H + MLP_H) g[P_B2 + t - MLP_OUT * MLP_H] = gc;
  else if (t < MLP_OUT * MLP_H + MLP_H + MLP_OUT) g[P_B3 + t - MLP_OUT * MLP_H - MLP_H] = gc;
  for (int o = 16; o > 0; o >>= 1) my_loss += __shfl_xor_sync(0xffffffffu, my_loss, o);
  if ((t & 31) == 0) S.loss[t >> 5] = my_loss;
  __syncthreads();
  if (t == 0) {
    float l = 0;
    for (int w = 0; w < GTHREADS / 32; ++w) l += S.loss[w];
    g[MLP_PARAMS] = l;
  }
}

struct AdamArgs {
  float *params, *m, *v;
  float lr, b1, b2, eps, c1, c2;
};

// The sum over the CTAs' parts, in CTA order within each of the block's 8
// warps (a warp every eighth part, a lane per parameter): into grad and *loss,
// or (ADAM) straight into an Adam step (Kingma & Ba 2015) on the FP32 master
// parameters, *loss then the mean over nb samples.
template <bool ADAM>
__global__ void __launch_bounds__(256) k_mlp_apply(const float *part, int parts, float *grad, float *loss,
                                                   AdamArgs a, float nb) {
  __shared__ float sum[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  float g = 0;
#pragma unroll 4
  for (int c = warp; c < parts; c += 8) g += part[(size_t)c * PART + k];
  sum[warp][lane] = g;
  __syncthreads();
  if (warp != 0 || k > MLP_PARAMS) return;
  g = 0;
  for (int w = 0; w < 8; ++w) g += sum[w][lane];
  if (k == MLP_PARAMS) {
    if (loss) *loss = ADAM ? __fdiv_rn(g, nb) : g;
    return;
  }
  if (!ADAM) {
    grad[k] = g;
    return;
  }
  const float mk = a.b1 * a.m[k] + (1 - a.b1) * g;
  const float vk = a.b2 * a.v[k] + (1 - a.b2) * g * g;
  a.m[k] = mk;
  a.v[k] = vk;
  a.params[k] -= a.lr * (mk / a.c1) / (sqrtf(vk / a.c2) + a.eps);
}

// The forward pass on CUDA cores (a thread per sample): the check of the
// tensor-core inference.
__global__ void k_mlp_infer_cc(const float *x, uint32_t n, const float *params, float *y) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float xi[MLP_IN], h1[MLP_H], h2[MLP_H];
  for (int k = 0; k < MLP_IN; ++k) xi[k] = bf(x[(size_t)i * MLP_IN + k]);
  for (int j = 0; j < MLP_H; ++j) {
    float z = params[P_B1 + j];
    for (int k = 0; k < MLP_IN; ++k) z += bf(params[P_W1 + j * MLP_IN + k]) * xi[k];
    h1[j] = bf(gelu(z));
  }
  for (int j = 0; j < MLP_H; ++j) {
    float z = params[P_B2 + j];
    for (int k = 0; k < MLP_H; ++k) z += bf(params[P_W2 + j * MLP_H + k]) * h1[k];
    h2[j] = bf(gelu(z));
  }
  for (int o = 0; o < MLP_OUT; ++o) {
    float z = params[P_B3 + o];
    for (int k = 0; k < MLP_H; ++k) z += bf(params[P_W3 + o * MLP_H + k]) * h2[k];
    y[(size_t)i * MLP_OUT + o] = z;
  }
}

}  // namespace

// ---- inference on the tensor cores ---------------------------------------------------------

// Shared memory of k_mlp_infer_tc: the operand tiles (bf16, K-major, the
// tile layout of tc.cuh) and the barriers.
struct InferSmem {
  unsigned char x[TT * 16 * 2];          // A1: 128 x 16 (12 inputs, zero padded)
  unsigned char h[TT * MLP_H * 2];       // A2 / A3: 128 x 64
  unsigned char w1[MLP_H * 16 * 2];      // B1: 64 (out) x 16 (in)
  unsigned char w2[MLP_H * MLP_H * 2];   // B2: 64 x 64
  unsigned char w3[16 * MLP_H * 2];      // B3: 16 (2 outputs, zero padded) x 64
  float b1[MLP_H], b2[MLP_H], b3[MLP_OUT];
  uint64_t bar;
  uint32_t tmem, err;
};

__device__ __forceinline__ void put_bf16(unsigned char *tile, uint32_t rows, uint32_t r, uint32_t k,
                                         float v) {
  *reinterpret_cast<__nv_bfloat16 *>(tile + tc::tile_offset(r, k / 8, rows) + (k % 8) * 2) =
      __float2bfloat16(v);
}

// y[i] = MLP(x[i]) for the 128 samples of this CTA's tile. x: n x 12 FP32;
// per-sample hook: rows with row_ok false produce nothing.
__global__ void __launch_bounds__(TT) k_mlp_infer_tc(const float *x, uint32_t n,
                                                     const float *params, float *y,
                                                     uint32_t *err_flag) {
  extern __shared__ __align__(1024) unsigned char mlp_tc_smem[];
  InferSmem &S = *reinterpret_cast<InferSmem *>(mlp_tc_smem);
  const uint32_t t = threadIdx.x, warp = t >> 5;
  const uint32_t i = blockIdx.x * TT + t;
  // operands: this thread's input row, and a share of the weight tiles
  for (uint32_t k = 0; k < 16; ++k)
    put_bf16(S.x, TT, t, k, (i < n && k < (uint32_t)MLP_IN) ? x[(size_t)i * MLP_IN + k] : 0.f);
  for (uint32_t e = t; e < MLP_H * 16; e += TT) {
    const uint32_t o = e / 16, k = e % 16;
    put_bf16(S.w1, MLP_H, o, k, k < (uint32_t)MLP_IN ? params[P_W1 + o * MLP_IN + k] : 0.f);
  }
  for (uint32_t e = t; e < MLP_H * MLP_H; e += TT)
    put_bf16(S.w2, MLP_H, e / MLP_H, e % MLP_H, params[P_W2 + e]);
  for (uint32_t e = t; e < 16 * MLP_H; e += TT) {
    const uint32_t o = e / MLP_H, k = e % MLP_H;
    put_bf16(S.w3, 16, o, k, o < (uint32_t)MLP_OUT ? params[P_W3 + o * MLP_H + k] : 0.f);
  }
  if (t < (uint32_t)MLP_H) {
    S.b1[t] = params[P_B1 + t];
    S.b2[t] = params[P_B2 + t];
  }
  if (t < (uint32_t)MLP_OUT) S.b3[t] = params[P_B3 + t];
  if (t == 0) {
    tc::mbar_init(&S.bar, 1);
    S.err = 0;
    tc::mbar_init_fence();
  }
  __syncwarp();
  if (warp == 0) {
    tc::tmem_alloc(&S.tmem, 128);
    tc::tmem_relinquish();
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = S.tmem;
  const uint32_t lane_base = (warp * 32u) << 16;
  volatile uint32_t *abort = &S.err;
  constexpr uint64_t BUDGET = 50ull * 1000 * 1000;
  const uint32_t hl = (TT / 8) * 128;  // LBO of the 128-row activation tiles
  bool ok = true;
  uint32_t phase = 0;
  // one layer: D (cols col0..) = A (rows TT, K = kdim) x B (rows nrows, K = kdim)
  auto layer = [&](const unsigned char *A, const unsigned char *B, uint32_t nrows, uint32_t kdim,
                   uint32_t col0) {
    if (t == 0) {
      tc::fence_after_sync();
      const uint32_t a0 = tc::smem_addr(A), b0 = tc::smem_addr(B), bl = (nrows / 8) * 128;
      const uint32_t idesc = tc::idesc_bf16_f32(TT, nrows);
      for (uint32_t ks = 0; ks < kdim / 16; ++ks)
        tc::mma_bf16(tmem + col0, tc::smem_desc(a0 + ks * 2 * hl, hl, 128),
                     tc::smem_desc(b0 + ks * 2 * bl, bl, 128), idesc, ks ? 1u : 0u);
      tc::commit(&S.bar);
    }
    if (!tc::mbar_wait(&S.bar, phase & 1, abort, BUDGET)) ok = false;
    ++phase;
    tc::fence_after_sync();
    ok = __syncthreads_and(ok);  // every thread of a warp takes the same path into tcgen05.ld
  };
  float v[32];
  // layer 1: x W1^T -> TMEM cols 0..63
  layer(S.x, S.w1, MLP_H, 16, 0);
  if (ok) {
    for (uint32_t c0 = 0; c0 < (uint32_t)MLP_H; c0 += 32) {
      tc::tmem_ld32(tmem + lane_base + c0, v);
      for (uint32_t k = 0; k < 32; ++k) put_bf16(S.h, TT, t, c0 + k, gelu(v[k] + S.b1[c0 + k]));
    }
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  // layer 2: h1 W2^T -> cols 64..127
  if (ok) layer(S.h, S.w2, MLP_H, MLP_H, 64);
  if (ok) {
    // the MMA has read h1 (its completion was waited on): h2 overwrites it
    for (uint32_t c0 = 0; c0 < (uint32_t)MLP_H; c0 += 32) {
      tc::tmem_ld32(tmem + lane_base + 64 + c0, v);
      for (uint32_t k = 0; k < 32; ++k) put_bf16(S.h, TT, t, c0 + k, gelu(v[k] + S.b2[c0 + k]));
    }
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  // layer 3: h2 W3^T -> cols 0..15
  if (ok) layer(S.h, S.w3, 16, MLP_H, 0);
  if (ok) {
    tc::tmem_ld32(tmem + lane_base, v);
    if (i < n)
      for (uint32_t o = 0; o < (uint32_t)MLP_OUT; ++o) y[(size_t)i * MLP_OUT + o] = v[o] + S.b3[o];
  }
  tc::fence_before_sync();
  const bool all_ok = __syncthreads_and(ok);
  if (warp == 0 && all_ok) tc::tmem_dealloc(tmem, 128);
  if (t == 0 && !all_ok && err_flag) atomicOr(err_flag, ST_WAIT_TIMEOUT);
}

int mlp_infer_tc(const float *x, uint32_t n, const float *params, float *y, uint32_t *err_flag,
                 cudaStream_t st) {
  if (n == 0) return 0;
  if (!open_shared<k_mlp_infer_tc>(sizeof(InferSmem))) return -1;
  D3_LAUNCH(k_mlp_infer_tc, blocks_for(n, TT), TT, sizeof(InferSmem), st)(x, n, params, y,
                                                                         err_flag);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace d3

using namespace d3;

namespace {

// CTAs of a gradient launch over n samples: a tile each, at most one an SM.
int grad_ctas(uint32_t n) {
  static int sms = 0;
  if (!sms) {
    int dev = 0, count = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    sms = count;
  }
  const unsigned b = blocks_for(n, GT);
  return b < (unsigned)sms ? (int)b : sms;
}

int grad_launch(const float *x, const float *y, uint32_t n, const float *params, float *part, int ctas,
                cudaStream_t st) {
  if (!open_shared<k_mlp_grad>(sizeof(TrainSmem))) return -1;
  D3_LAUNCH(k_mlp_grad, ctas, GTHREADS, sizeof(TrainSmem), st)(x, y, n, params, (float)n, part);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

constexpr unsigned APPLY_BLOCKS = PART / 32;

}  // namespace

extern "C" int32_t d3_mlp_grad(const float *x, const float *y, uint32_t n, const float *params,
                               float *grad, float *loss) {
  if (!x || !y || !params || !grad || !loss || n == 0) return D3_BAD_ARGUMENT;
  const int ctas = grad_ctas(n);
  float *d = nullptr;
  if (cudaMalloc(&d, (2 * MLP_PARAMS + 1 + (size_t)ctas * PART) * 4) != cudaSuccess) return D3_OUT_OF_MEMORY;
  float *dp = d, *dg = d + MLP_PARAMS, *dl = d + 2 * MLP_PARAMS, *part = dl + 1;
  int32_t rc = D3_OK;
  if (cudaMemcpy(dp, params, MLP_PARAMS * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      grad_launch(x, y, n, dp, part, ctas, 0))
    rc = D3_WORKER_FAILED;
  if (rc == D3_OK) {
    D3_LAUNCH(k_mlp_apply<false>, APPLY_BLOCKS, 256, 0, 0)(part, ctas, dg, dl, AdamArgs{}, 1.f);
    if (cudaMemcpy(grad, dg, MLP_PARAMS * 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(loss, dl, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = D3_WORKER_FAILED;
  }
  *loss /= (float)n;
  cudaFree(d);
  return rc;
}

extern "C" int32_t d3_mlp_train(const float *x, const float *y, uint32_t n, uint32_t batch,
                                uint32_t steps, float lr, float *params, float *losses) {
  if (!x || !y || !params || n == 0 || batch == 0) return D3_BAD_ARGUMENT;
  const uint32_t nb = batch < n ? batch : n;
  const int ctas = grad_ctas(nb);
  float *d = nullptr;
  if (cudaMalloc(&d, (3 * MLP_PARAMS + (size_t)ctas * PART + steps) * 4) != cudaSuccess)
    return D3_OUT_OF_MEMORY;
  float *dp = d, *dm = d + MLP_PARAMS, *dv = d + 2 * MLP_PARAMS, *part = d + 3 * MLP_PARAMS,
        *dl = part + (size_t)ctas * PART;
  int32_t rc = D3_OK;
  cudaStream_t st = 0;
  if (cudaMemcpy(dp, params, MLP_PARAMS * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(dm, 0, 2 * MLP_PARAMS * 4) != cudaSuccess)
    rc = D3_WORKER_FAILED;
  AdamArgs a{dp, dm, dv, lr, 0.9f, 0.999f, 1e-8f, 0, 0};
  float c1 = 1, c2 = 1;
  uint32_t off = 0;
  for (uint32_t s = 0; s < steps && rc == D3_OK; ++s) {
    if (off + nb > n) off = 0;  // batches walk the (pre-shuffled) samples in order
    if (grad_launch(x + (size_t)off * MLP_IN, y + (size_t)off * MLP_OUT, nb, dp, part, ctas, st)) {
      rc = D3_WORKER_FAILED;
      break;
    }
    off += nb;
    c1 *= a.b1;
    c2 *= a.b2;
    a.c1 = 1 - c1;
    a.c2 = 1 - c2;
    D3_LAUNCH(k_mlp_apply<true>, APPLY_BLOCKS, 256, 0, st)(part, ctas, nullptr, dl + s, a, (float)nb);
  }
  // the step losses come back once, with the parameters
  if (rc == D3_OK && (cudaMemcpy(params, dp, MLP_PARAMS * 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
                      (losses && steps &&
                       cudaMemcpy(losses, dl, steps * 4ull, cudaMemcpyDeviceToHost) != cudaSuccess)))
    rc = D3_WORKER_FAILED;
  cudaFree(d);
  return rc;
}

extern "C" int32_t d3_mlp_infer(const float *x, uint32_t n, const float *params, float *y,
                                uint32_t tensor_cores) {
  if (!x || !params || !y) return D3_BAD_ARGUMENT;
  float *dp = nullptr;
  uint32_t *flag = nullptr;
  if (cudaMalloc(&dp, MLP_PARAMS * 4) != cudaSuccess || cudaMalloc(&flag, 4) != cudaSuccess) {
    cudaFree(dp);
    return D3_OUT_OF_MEMORY;
  }
  int32_t rc = D3_OK;
  uint32_t h_flag = 0;
  if (cudaMemcpy(dp, params, MLP_PARAMS * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(flag, 0, 4) != cudaSuccess)
    rc = D3_WORKER_FAILED;
  if (rc == D3_OK) {
    if (tensor_cores) {
      if (mlp_infer_tc(x, n, dp, y, flag, 0)) rc = D3_WORKER_FAILED;
    } else {
      D3_LAUNCH(k_mlp_infer_cc, blocks_for(n, 128), 128, 0, 0)(x, n, dp, y);
    }
  }
  if (cudaMemcpy(&h_flag, flag, 4, cudaMemcpyDeviceToHost) != cudaSuccess || h_flag)
    rc = D3_WORKER_FAILED;
  cudaFree(dp);
  cudaFree(flag);
  return rc;
}
