// bl_mlp.cu -- the learned mixed-cell closure's network: 10 inputs, two
// hidden layers of 64 with SiLU, 2 outputs, trained and evaluated on the
// tensor cores (BF16 operands, FP32 accumulation) by the kernels below.
//
//   z1 = W1 x + b1, h1 = silu(z1), z2 = W2 h1 + b2, h2 = silu(z2),
//   y = W3 h2 + b3,  loss = sum over samples and outputs of (y - t)^2 / (2 n)
//
// Every product of the forward and backward passes is a 16x8x16 tile
// product (mma.sync m16n8k16, BF16 x BF16 -> FP32) of 16 samples per warp:
// the activations and weights are rounded to BF16 where they enter a
// product, everything else (biases, SiLU, sums, Adam) stays FP32.  The
// weight gradients of a block of 64 samples are summed on the tensor cores
// too (the sample dimension is the product's k), then over blocks in a
// fixed order, so training is deterministic.  Parameters are FP32 master
// copies in one array (layout below); no CPU path exists.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/bookleaf_gb300.h"
#include "bl_mma.cuh"

namespace {

using namespace bl::mlp;

__device__ void load_x(SmemS& s, const float* X, int base, int n) {
  for (int i = threadIdx.x & 31; i < 16 * 16; i += 32) {
    const int r = i / 16, c = i % 16, row = base + r;
    s.x[r][c] = (c < NI && row < n) ? X[(size_t)row * NI + c] : 0.0f;
  }
  __syncwarp();
}

__global__ void __launch_bounds__(TPB) k_mlp_forward(const float* img, const float* X, float* Y,
                                                     int n) {
  extern __shared__ unsigned char smem[];
  SmemW& w = *reinterpret_cast<SmemW*>(smem);
  SmemS* S = reinterpret_cast<SmemS*>(smem + sizeof(SmemW));
  copy_weights<TPB>(w, img);
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  SmemS& s = S[warp];
  const int base = blockIdx.x * SPB + warp * 16;
  load_x(s, X, base, n);
  forward_warp(w, s);
  for (int i = threadIdx.x & 31; i < 16 * NO; i += 32) {
    const int r = i / NO, c = i % NO;
    if (base + r < n) Y[(size_t)(base + r) * NO + c] = s.y[r][c];
  }
}

// ---------------------------------------------------------------- gradient
//
// Forward and backward of one block's 64 samples and their gradient sum, by
// 8 warps.  Everything that enters a product is held in shared memory as
// the BF16 it is rounded to, in rows padded by 16 bytes, and read as whole
// fragments (ldmatrix, transposed where a product runs over the samples or
// against a weight's rows); warp w takes samples 16 (w & 3) .. + 16 of each
// layer and half w >> 2 of its outputs, whose pre-activations and sigmoids
// stay in the accumulators' registers for the backward pass.  The products,
// their order of accumulation and the FP32 arithmetic between them are those
// of the version that kept FP32 in shared memory and packed every operand
// anew (30 us for one block, nearly all of it shared-memory loads and
// conversions; about 3.5 us so).
constexpr int GW = 8, GT = 32 * GW;    // warps, threads of a gradient block
constexpr int PX = 24, PH = 72, PF = 68;  // padded rows: 16 and 64 BF16, 64 FP32
struct SmemG {
  // weights as BF16, biases FP32
  __nv_bfloat16 w1[NH][PX], w2[NH][PH], w3[16][PH];
  float b1[NH], b2[NH], b3[16];
  // samples, activations and their gradients as BF16
  __nv_bfloat16 x[SPB][PX], dy[SPB][PX];
  __nv_bfloat16 h1[SPB][PH], h2[SPB][PH], dz1[SPB][PH], dz2[SPB][PH];
  // FP32 for the bias sums
  float dz1f[SPB][PF], dz2f[SPB][PF], dyf[SPB][NO];
  float t[SPB][NO];
  float lsum[GW], loss;
  float g[NP];  // the block's gradient, in the parameters' layout
};

__device__ __forceinline__ uint32_t smem_at(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldm2(uint32_t (&r)[2], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldm2t(uint32_t (&r)[2], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(smem_at(p)) : "memory");
}
// A (16 x 16) = rows r0.., columns c0.. of a row-major array
template <int P>
__device__ __forceinline__ void a_rows(uint32_t (&r)[4], const __nv_bfloat16 (*m)[P], int r0, int c0) {
  const int l = threadIdx.x & 31;
  ldm4(r, &m[r0 + (l & 15)][c0 + ((l >> 4) << 3)]);
}
// A (16 x 16) = the transpose of rows k0.., columns r0..
template <int P>
__device__ __forceinline__ void a_cols(uint32_t (&r)[4], const __nv_bfloat16 (*m)[P], int k0, int r0) {
  const int l = threadIdx.x & 31;
  ldm4t(r, &m[k0 + ((l >> 4) << 3) + (l & 7)][r0 + (((l >> 3) & 1) << 3)]);
}
// B (16 x 8), b(k, n) = m[n0 + n][k0 + k]
template <int P>
__device__ __forceinline__ void b_rows(uint32_t (&r)[2], const __nv_bfloat16 (*m)[P], int n0, int k0) {
  const int l = threadIdx.x & 31;
  ldm2(r, &m[n0 + (l & 7)][k0 + (((l >> 3) & 1) << 3)]);
}
// B (16 x 8), b(k, n) = m[k0 + k][n0 + n]
template <int P>
__device__ __forceinline__ void b_cols(uint32_t (&r)[2], const __nv_bfloat16 (*m)[P], int k0, int n0) {
  const int l = threadIdx.x & 31;
  ldm2t(r, &m[k0 + (l & 15)][n0]);
}
__device__ __forceinline__ void put2(__nv_bfloat16* p, float lo, float hi) {
  *reinterpret_cast<uint32_t*>(p) = pack(lo, hi);
}

// where parameter i stands among the weights of a gradient block
struct Place {
  void* at;
  bool bias;  // FP32, else BF16
};
__device__ __forceinline__ Place place_of(SmemG& s, int i) {
  if (i < OB1) return {&s.w1[i / NI][i % NI], false};
  if (i < OW2) return {&s.b1[i - OB1], true};
  if (i < OB2) return {&s.w2[(i - OW2) / NH][(i - OW2) % NH], false};
  if (i < OW3) return {&s.b2[i - OB2], true};
  if (i < OB3) return {&s.w3[(i - OW3) / NH][(i - OW3) % NH], false};
  return {&s.b3[i - OB3], true};
}
// zero padding (once per block), then every parameter from P
__device__ void load_params(SmemG& s, const float* P) {
  for (int i = threadIdx.x; i < NH * PX; i += GT) (&s.w1[0][0])[i] = __float2bfloat16_rn(0.0f);
  for (int i = threadIdx.x; i < 16 * PH; i += GT) (&s.w3[0][0])[i] = __float2bfloat16_rn(0.0f);
  for (int i = threadIdx.x; i < SPB * PX; i += GT) {
    (&s.x[0][0])[i] = __float2bfloat16_rn(0.0f);
    (&s.dy[0][0])[i] = __float2bfloat16_rn(0.0f);
  }
  if (threadIdx.x < 16) s.b3[threadIdx.x] = 0.0f;
  __syncthreads();
  for (int i = threadIdx.x; i < NP; i += GT) {
    const Place w = place_of(s, i);
    if (w.bias) *static_cast<float*>(w.at) = P[i];
    else *static_cast<__nv_bfloat16*>(w.at) = __float2bfloat16_rn(P[i]);
  }
}

// A block's samples in flight: thread i holds inputs i, i + GT, ... of the
// 64 x 10 and target i of the 64 x 2.
constexpr int XPT = (SPB * NI + GT - 1) / GT;
struct Fetched {
  float x[XPT], t;
};
__device__ __forceinline__ Fetched fetch_samples(const float* X, const float* T, const int* idx,
                                                 int base, int n) {
  Fetched f;
#pragma unroll
  for (int k = 0; k < XPT; k++) {
    const int i = threadIdx.x + k * GT, r = i / NI, row = base + r;
    f.x[k] = 0.0f;
    if (r < SPB && row < n) f.x[k] = __ldg(X + (size_t)(idx ? __ldg(idx + row) : row) * NI + i % NI);
  }
  f.t = 0.0f;
  if (threadIdx.x < SPB * NO) {
    const int row = base + (int)threadIdx.x / NO;
    if (row < n)
      f.t = __ldg(T + (size_t)(idx ? __ldg(idx + row) : row) * NO + threadIdx.x % NO);
  }
  return f;
}
__device__ __forceinline__ void place_samples(SmemG& s, const Fetched& f) {
#pragma unroll
  for (int k = 0; k < XPT; k++) {
    const int i = threadIdx.x + k * GT;
    if (i < SPB * NI) s.x[i / NI][i % NI] = __float2bfloat16_rn(f.x[k]);
  }
  if (threadIdx.x < SPB * NO) s.t[threadIdx.x / NO][threadIdx.x % NO] = f.t;
}

// s.g = the sum over the block's samples (rows base + r < n) of the
// gradient, s.loss its loss share; s.x, s.t and the weights are in place
// (a barrier behind them).  Ends with a barrier.
__device__ __forceinline__ void block_gradient(SmemG& s, int base, int n, float inv_n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
  uint32_t a[4], b[2];
  float z1[4][4], s1[4][4], z2[4][4], s2[4][4];
  // layer 1: z1 = x W1^T + b1
  a_rows(a, s.x, r0, 0);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    float d[4] = {0, 0, 0, 0};
    b_rows(b, s.w1, n0 + q * 8, 0);
    mma16816(d, a, b);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      z1[q][i] = d[i] + s.b1[n0 + q * 8 + 2 * t + (i & 1)];
      s1[q][i] = sigm(z1[q][i]);
    }
    put2(&s.h1[r0 + g][n0 + q * 8 + 2 * t], z1[q][0] * s1[q][0], z1[q][1] * s1[q][1]);
    put2(&s.h1[r0 + g + 8][n0 + q * 8 + 2 * t], z1[q][2] * s1[q][2], z1[q][3] * s1[q][3]);
  }
  __syncthreads();
  // layer 2: z2 = h1 W2^T + b2
  {
    float d[4][4] = {};
#pragma unroll
    for (int kt = 0; kt < NH / 16; kt++) {
      a_rows(a, s.h1, r0, kt * 16);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        b_rows(b, s.w2, n0 + q * 8, kt * 16);
        mma16816(d[q], a, b);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        z2[q][i] = d[q][i] + s.b2[n0 + q * 8 + 2 * t + (i & 1)];
        s2[q][i] = sigm(z2[q][i]);
      }
      put2(&s.h2[r0 + g][n0 + q * 8 + 2 * t], z2[q][0] * s2[q][0], z2[q][1] * s2[q][1]);
      put2(&s.h2[r0 + g + 8][n0 + q * 8 + 2 * t], z2[q][2] * s2[q][2], z2[q][3] * s2[q][3]);
    }
  }
  __syncthreads();
  // layer 3 and dy = (y - t) / n for valid samples; loss terms (warps 0-3;
  // lanes t = 0 hold the two outputs)
  if (warp < 4) {
    float d[4] = {0, 0, 0, 0};
#pragma unroll
    for (int kt = 0; kt < NH / 16; kt++) {
      a_rows(a, s.h2, r0, kt * 16);
      b_rows(b, s.w3, 0, kt * 16);
      mma16816(d, a, b);
    }
    float lp = 0.0f;
    if (t == 0) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = r0 + g + 8 * h;
        float e0 = d[2 * h] + s.b3[0] - s.t[r][0], e1 = d[2 * h + 1] + s.b3[1] - s.t[r][1];
        if (base + r >= n) e0 = e1 = 0.0f;
        lp += e0 * e0 + e1 * e1;
        e0 = e0 * inv_n;
        e1 = e1 * inv_n;
        s.dyf[r][0] = e0;
        s.dyf[r][1] = e1;
        put2(&s.dy[r][0], e0, e1);
      }
    }
    for (int o = 16; o > 0; o >>= 1) lp += __shfl_xor_sync(0xffffffffu, lp, o);
    if (lane == 0) s.lsum[warp] = lp;
  }
  __syncthreads();
  // dh2 = dy W3 (K = 16 padded outputs); dz2 = dh2 silu'(z2)
  a_rows(a, s.dy, r0, 0);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    float d[4] = {0, 0, 0, 0};
    b_cols(b, s.w3, 0, n0 + q * 8);
    mma16816(d, a, b);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float z = z2[q][i], sg = s2[q][i];
      d[i] = d[i] * sg * (1.0f + z * (1.0f - sg));
    }
    const int c = n0 + q * 8 + 2 * t;
    put2(&s.dz2[r0 + g][c], d[0], d[1]);
    put2(&s.dz2[r0 + g + 8][c], d[2], d[3]);
    *reinterpret_cast<float2*>(&s.dz2f[r0 + g][c]) = make_float2(d[0], d[1]);
    *reinterpret_cast<float2*>(&s.dz2f[r0 + g + 8][c]) = make_float2(d[2], d[3]);
  }
  __syncthreads();
  // dh1 = dz2 W2; dz1 = dh1 silu'(z1)
  {
    float d[4][4] = {};
#pragma unroll
    for (int kt = 0; kt < NH / 16; kt++) {
      a_rows(a, s.dz2, r0, kt * 16);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        b_cols(b, s.w2, kt * 16, n0 + q * 8);
        mma16816(d[q], a, b);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float z = z1[q][i], sg = s1[q][i];
        d[q][i] = d[q][i] * sg * (1.0f + z * (1.0f - sg));
      }
      const int c = n0 + q * 8 + 2 * t;
      put2(&s.dz1[r0 + g][c], d[q][0], d[q][1]);
      put2(&s.dz1[r0 + g + 8][c], d[q][2], d[q][3]);
      *reinterpret_cast<float2*>(&s.dz1f[r0 + g][c]) = make_float2(d[q][0], d[q][1]);
      *reinterpret_cast<float2*>(&s.dz1f[r0 + g + 8][c]) = make_float2(d[q][2], d[q][3]);
    }
  }
  __syncthreads();
  // Weight gradients summed over the block's 64 samples (the k of the
  // products): dW = dZ^T A with A the layer's input activations.  Warp w
  // takes the output rows 16 (w & 3) .. of dW1 and dW2 and half the columns
  // of each, and 8 columns of dW3.
  {
    float d[4][4] = {}, e[4] = {0, 0, 0, 0}, f[4] = {0, 0, 0, 0};
#pragma unroll
    for (int kt = 0; kt < SPB / 16; kt++) {
      a_cols(a, s.dz2, kt * 16, r0);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        b_cols(b, s.h1, kt * 16, n0 + q * 8);
        mma16816(d[q], a, b);
      }
      a_cols(a, s.dz1, kt * 16, r0);
      b_cols(b, s.x, kt * 16, (warp >> 2) * 8);
      mma16816(e, a, b);
      a_cols(a, s.dy, kt * 16, 0);
      b_cols(b, s.h2, kt * 16, warp * 8);
      mma16816(f, a, b);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int o = r0 + g + 8 * (i >> 1), c = 2 * t + (i & 1);
#pragma unroll
      for (int q = 0; q < 4; q++) s.g[OW2 + o * NH + n0 + q * 8 + c] = d[q][i];
      const int c1 = (warp >> 2) * 8 + c;
      if (c1 < NI) s.g[OW1 + o * NI + c1] = e[i];
      const int o3 = g + 8 * (i >> 1);
      if (o3 < NO) s.g[OW3 + o3 * NH + warp * 8 + c] = f[i];
    }
  }
  // bias gradients: column sums over the block's samples (FP32)
  if (threadIdx.x < 2 * NH) {
    const int i = threadIdx.x & (NH - 1);
    const float(*z)[PF] = threadIdx.x < NH ? s.dz1f : s.dz2f;
    float v = 0.0f;
#pragma unroll 16
    for (int r = 0; r < SPB; r++) v += z[r][i];
    s.g[(threadIdx.x < NH ? OB1 : OB2) + i] = v;
  } else if (threadIdx.x < 2 * NH + NO) {
    const int i = threadIdx.x - 2 * NH;
    float v = 0.0f;
#pragma unroll 16
    for (int r = 0; r < SPB; r++) v += s.dyf[r][i];
    s.g[OB3 + i] = v;
  } else if (threadIdx.x == GT - 1) {
    s.loss = 0.5f * inv_n * (s.lsum[0] + s.lsum[1] + s.lsum[2] + s.lsum[3]);
  }
  __syncthreads();
}

// One block's 64 samples; its gradient sum and loss share go to
// G[blockIdx][NP] and L[blockIdx].
__global__ void __launch_bounds__(GT) k_mlp_grad(const float* P, const float* X, const float* T,
                                                 const int* idx, int n, float inv_n, float* G,
                                                 float* L) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmemG& s = *reinterpret_cast<SmemG*>(smem);
  const int base = blockIdx.x * SPB;
  const Fetched f = fetch_samples(X, T, idx, base, n);
  load_params(s, P);
  place_samples(s, f);
  __syncthreads();
  block_gradient(s, base, n, inv_n);
  for (int i = threadIdx.x; i < NP; i += GT) G[(size_t)blockIdx.x * NP + i] = s.g[i];
  if (threadIdx.x == 0) L[blockIdx.x] = s.loss;
}

// Adam on one FP32 master parameter (Kingma and Ba, 2015), c1 and c2 the
// bias corrections of the update
struct AdamStep {
  float p, m, v;
};
__device__ __forceinline__ AdamStep adam(float P, float M, float V, float g, float lr, float b1,
                                         float b2, float eps, float c1, float c2) {
  const float m = b1 * M + (1.0f - b1) * g, v = b2 * V + (1.0f - b2) * g * g;
  return {P - lr * (m * c1) / (sqrtf(v * c2) + eps), m, v};
}

// A whole epoch of mini-batches of up to 8 blocks in one launch: one thread
// block cluster, a block per 64 samples, everything on chip.  Per
// mini-batch each block forms its gradient in its shared memory; the blocks
// then each sum a share of the parameters over the cluster (in block order,
// through distributed shared memory), take Adam's step on it (the share's
// master copies and moments stay with it for the epoch) and write the new
// weights into every block's BF16 copy.  The next mini-batch's samples are
// fetched meanwhile.  Launched one by one, gradient, sum and Adam took 28.6
// us a mini-batch of 256; so it takes 7.5 us, of which the gradient 3.4, Adam
// and the exchange 2.5 and the cluster's barriers 1.1.
constexpr int kMaxCluster = 8;
struct EpochArgs {
  float *P, *M, *V, *img;
  const float *X, *T;
  const int* idx;
  int n, batch;
  float lr, b1, b2, eps;
  const float *c1t, *c2t;  // this epoch's bias corrections
  double* acc;             // the epoch's loss sum
};
__host__ __device__ constexpr int epoch_share(int nb) { return (NP + nb - 1) / nb; }
inline size_t epoch_smem(int nb) {
  return sizeof(SmemG) + 3 * sizeof(float) * (size_t)epoch_share(nb);
}
__global__ void __launch_bounds__(GT) k_mlp_epoch(EpochArgs A) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem[];
  SmemG& s = *reinterpret_cast<SmemG*>(smem);
  cg::cluster_group cl = cg::this_cluster();
  const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int share = epoch_share(nb), p0 = rank * share, p1 = min(p0 + share, (int)NP);
  float* const pS = reinterpret_cast<float*>(smem + sizeof(SmemG));
  float* const mS = pS + share;
  float* const vS = mS + share;
  Fetched f = fetch_samples(A.X, A.T, A.idx, rank * SPB, min(A.batch, A.n));
  load_params(s, A.P);
  for (int i = p0 + threadIdx.x; i < p1; i += GT) {
    pS[i - p0] = A.P[i];
    mS[i - p0] = A.M[i];
    vS[i - p0] = A.V[i];
  }
  double acc = 0.0;
  const int nbat = (A.n + A.batch - 1) / A.batch;
  for (int k = 0; k < nbat; k++) {
    const int size = min(A.batch, A.n - k * A.batch);  // samples of this mini-batch
    const int blocks = (size + SPB - 1) / SPB;
    place_samples(s, f);
    __syncthreads();
    if (k + 1 < nbat)
      f = fetch_samples(A.X, A.T, A.idx + (size_t)(k + 1) * A.batch, rank * SPB,
                        min(A.batch, A.n - (k + 1) * A.batch));
    const float c1 = __ldg(A.c1t + k), c2 = __ldg(A.c2t + k);
    if (rank < blocks) block_gradient(s, rank * SPB, size, 1.0f / (float)size);
    cl.sync();
    // two parameters a turn, their shares of every block asked for at once
    for (int i0 = p0 + threadIdx.x; i0 < p1; i0 += 2 * GT) {
      float q[2][kMaxCluster];
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int b = 0; b < kMaxCluster; b++) {
          const int i = i0 + j * GT;
          q[j][b] = i < p1 && b < blocks ? *cl.map_shared_rank(&s.g[i], b) : 0.0f;
        }
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int i = i0 + j * GT;
        if (i >= p1) break;
        float g = 0.0f;
#pragma unroll
        for (int b = 0; b < kMaxCluster; b++)
          if (b < blocks) g += q[j][b];
        const AdamStep u = adam(pS[i - p0], mS[i - p0], vS[i - p0], g, A.lr, A.b1, A.b2, A.eps, c1, c2);
        pS[i - p0] = u.p;
        mS[i - p0] = u.m;
        vS[i - p0] = u.v;
        const Place w = place_of(s, i);
        if (w.bias) {
          for (int b = 0; b < nb; b++) *cl.map_shared_rank(static_cast<float*>(w.at), b) = u.p;
        } else {
          const __nv_bfloat16 h = __float2bfloat16_rn(u.p);
          for (int b = 0; b < nb; b++) *cl.map_shared_rank(static_cast<__nv_bfloat16*>(w.at), b) = h;
        }
      }
    }
    if (rank == 0 && threadIdx.x == 0) {
      float l = 0.0f;
      for (int b = 0; b < blocks; b++) l += *cl.map_shared_rank(&s.loss, b);
      acc += (double)l * size;
    }
    cl.sync();
  }
  for (int i = p0 + threadIdx.x; i < p1; i += GT) {
    A.P[i] = pS[i - p0];
    A.M[i] = mS[i - p0];
    A.V[i] = vS[i - p0];
    A.img[image_offset(i)] = pS[i - p0];
  }
  if (rank == 0 && threadIdx.x == 0) *A.acc = acc;
}

// Sums the per-block gradients and losses in block order; the loss times
// wgt is also added to *acc (an epoch's running sum), in launch order.
__global__ void k_mlp_reduce(const float* G, const float* L, int nblk, float* grad, float* loss,
                             double* acc, double wgt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NP) {
    float s = 0.0f;
    for (int b = 0; b < nblk; b++) s += G[(size_t)b * NP + i];
    grad[i] = s;
  }
  if (i == 0) {
    float s = 0.0f;
    for (int b = 0; b < nblk; b++) s += L[b];
    *loss = s;
    if (acc) *acc += (double)s * wgt;
  }
}

// The parameters' shared-memory image (its padding is zeroed once).
__global__ void k_mlp_image(const float* P, float* img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NP) img[image_offset(i)] = P[i];
}

// Adam on every parameter, for mini-batches too large for one cluster; the
// image is kept current with the parameters.  The bias corrections of this
// update are entry *ebase + k of the tables c1t, c2t (the mini-batch k of an
// epoch whose first update is *ebase), so that one captured epoch replays
// with the next epoch's values.
__global__ void k_mlp_adam(float* P, float* M, float* V, float* img, const float* grad, float lr,
                           float b1, float b2, float eps, const float* c1t, const float* c2t,
                           const int* ebase, int k) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NP) return;
  const float c1 = c1t[*ebase + k], c2 = c2t[*ebase + k];
  const float g = grad[i];
  const float m = b1 * M[i] + (1.0f - b1) * g, v = b2 * V[i] + (1.0f - b2) * g * g;
  M[i] = m;
  V[i] = v;
  const float p = P[i] - lr * (m * c1) / (sqrtf(v * c2) + eps);
  P[i] = p;
  img[image_offset(i)] = p;
}

constexpr size_t kSmemFwd = sizeof(SmemW) + WARPS * sizeof(SmemS);
constexpr size_t kSmemGrad = sizeof(SmemG);

}  // namespace

struct bl_mlp {
  float *P = nullptr, *M = nullptr, *V = nullptr, *grad = nullptr, *loss = nullptr;
  float* img = nullptr;  // SmemW image of P
  double* acc = nullptr;  // an epoch's loss sum
  int step = 0;
};

extern "C" {

int bl_mlp_create(bl_mlp** out, const float* params) {
  if (!out || !params) return BL_FAILURE;
  *out = nullptr;
  bl_mlp* m = new bl_mlp();
  bool ok = cudaMalloc(&m->P, NP * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->M, NP * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->V, NP * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->grad, NP * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->loss, sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->img, kImgN * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&m->acc, sizeof(double)) == cudaSuccess;
  ok = ok && cudaMemcpy(m->P, params, NP * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess &&
       cudaMemset(m->M, 0, NP * sizeof(float)) == cudaSuccess &&
       cudaMemset(m->V, 0, NP * sizeof(float)) == cudaSuccess &&
       cudaMemset(m->img, 0, kImgN * sizeof(float)) == cudaSuccess;
  if (ok) {
    k_mlp_image<<<(NP + 255) / 256, 256>>>(m->P, m->img);
    ok = cudaDeviceSynchronize() == cudaSuccess;
  }
  ok = ok && cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kSmemFwd) == cudaSuccess &&
       cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kSmemGrad) == cudaSuccess &&
       cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)epoch_smem(1)) == cudaSuccess;
  if (!ok) {
    bl_mlp_destroy(m);
    return BL_FAILURE;
  }
  *out = m;
  return BL_SUCCESS;
}

int bl_mlp_destroy(bl_mlp* m) {
  if (!m) return BL_SUCCESS;
  cudaFree(m->P);
  cudaFree(m->M);
  cudaFree(m->V);
  cudaFree(m->grad);
  cudaFree(m->loss);
  cudaFree(m->img);
  cudaFree(m->acc);
  delete m;
  return BL_SUCCESS;
}

int bl_mlp_params(bl_mlp* m, float* params) {
  if (!m || !params) return BL_FAILURE;
  return cudaMemcpy(params, m->P, NP * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
             ? BL_SUCCESS : BL_FAILURE;
}

// The device image of the current parameters (the layout the closure
// kernel copies into shared memory); bl_set_closure takes a copy.
const float* bl_mlp_device_image(bl_mlp* m) { return m ? m->img : nullptr; }

int bl_mlp_predict(bl_mlp* m, const float* x, int n, float* y) {
  if (!m || !x || !y || n < 0) return BL_FAILURE;
  if (n == 0) return BL_SUCCESS;
  float *dx = nullptr, *dy = nullptr;
  bool ok = cudaMalloc(&dx, (size_t)n * NI * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&dy, (size_t)n * NO * sizeof(float)) == cudaSuccess;
  ok = ok && cudaMemcpy(dx, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_mlp_forward<<<(n + SPB - 1) / SPB, TPB, kSmemFwd>>>(m->img, dx, dy, n);
    ok = cudaMemcpy(y, dy, (size_t)n * NO * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(dx);
  cudaFree(dy);
  return ok ? BL_SUCCESS : BL_FAILURE;
}

int bl_mlp_gradient(bl_mlp* m, const float* x, const float* t, int n, float* grad, float* loss) {
  if (!m || !x || !t || !grad || n < 1) return BL_FAILURE;
  const int nblk = (n + SPB - 1) / SPB;
  float *dx = nullptr, *dt = nullptr, *G = nullptr, *L = nullptr;
  bool ok = cudaMalloc(&dx, (size_t)n * NI * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&dt, (size_t)n * NO * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&G, (size_t)nblk * NP * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&L, (size_t)nblk * sizeof(float)) == cudaSuccess;
  ok = ok && cudaMemcpy(dx, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess &&
       cudaMemcpy(dt, t, (size_t)n * NO * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_mlp_grad<<<nblk, GT, kSmemGrad>>>(m->P, dx, dt, nullptr, n, 1.0f / (float)n, G, L);
    k_mlp_reduce<<<(NP + 255) / 256, 256>>>(G, L, nblk, m->grad, m->loss, nullptr, 0.0);
    ok = cudaMemcpy(grad, m->grad, NP * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess;
    if (ok && loss) ok = cudaMemcpy(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(dx);
  cudaFree(dt);
  cudaFree(G);
  cudaFree(L);
  return ok ? BL_SUCCESS : BL_FAILURE;
}

int bl_mlp_train(bl_mlp* m, const float* x, const float* t, int n, int epochs, int batch,
                 float lr, unsigned long long seed, float* losses) {
  if (!m || !x || !t || n < 1 || epochs < 1 || batch < SPB) return BL_FAILURE;
  const int nb_per = (std::min(batch, n) + SPB - 1) / SPB;
  const int nbat = (n + batch - 1) / batch;  // mini-batches per epoch
  const long nupd = (long)epochs * nbat;
  const bool cluster = nb_per <= kMaxCluster;
  // one allocation: samples, two epochs' orders, bias corrections, the
  // epochs' loss sums (and the large mini-batches' block sums)
  size_t total = 0;
  auto part = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t ox = part((size_t)n * NI * sizeof(float)), ot = part((size_t)n * NO * sizeof(float)),
               oi = part(2 * (size_t)n * sizeof(int)), o1 = part((size_t)nupd * sizeof(float)),
               o2 = part((size_t)nupd * sizeof(float)), oa = part((size_t)epochs * sizeof(double)),
               oe = part(sizeof(int)), og = part(cluster ? 0 : (size_t)nb_per * NP * sizeof(float)),
               ol = part(cluster ? 0 : (size_t)nb_per * sizeof(float));
  char* mem = nullptr;
  bool ok = cudaMalloc(&mem, total) == cudaSuccess;
  float *dx = reinterpret_cast<float*>(mem + ox), *dt = reinterpret_cast<float*>(mem + ot);
  float *c1t = reinterpret_cast<float*>(mem + o1), *c2t = reinterpret_cast<float*>(mem + o2);
  float *G = reinterpret_cast<float*>(mem + og), *L = reinterpret_cast<float*>(mem + ol);
  int *didx = reinterpret_cast<int*>(mem + oi), *ebase = reinterpret_cast<int*>(mem + oe);
  double* acc = reinterpret_cast<double*>(mem + oa);
  ok = ok && cudaMemcpy(dx, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess &&
       cudaMemcpy(dt, t, (size_t)n * NO * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  // Adam's bias corrections for every update of the run (update u has step
  // count m->step + 1 + u)
  if (ok) {
    std::vector<float> c1(nupd), c2(nupd);
    for (long u = 0; u < nupd; u++) {
      const float st = (float)(m->step + 1 + u);
      c1[u] = 1.0f / (1.0f - powf(b1, st));
      c2[u] = 1.0f / (1.0f - powf(b2, st));
    }
    ok = cudaMemcpy(c1t, c1.data(), nupd * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(c2t, c2.data(), nupd * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
  }
  // cs runs the epochs, up brings each epoch's order while the one before
  // runs; done[e & 1] marks the end of epoch e, whose order buffer the
  // epoch after next takes
  cudaStream_t cs = nullptr, up = nullptr;
  cudaEvent_t done[2] = {nullptr, nullptr};
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  // (cs follows the copies and kernels of the legacy stream)
  ok = ok && cudaStreamCreate(&cs) == cudaSuccess &&
       cudaStreamCreateWithFlags(&up, cudaStreamNonBlocking) == cudaSuccess;
  for (auto& e : done) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (ok && !cluster) {
    // mini-batches beyond one cluster: an epoch's launches captured once as
    // a graph that reads the first order buffer
    ok = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    for (int k = 0; k < nbat && ok; k++) {
      const int b0 = k * batch, nb = std::min(batch, n - b0);
      const int nblk = (nb + SPB - 1) / SPB;
      k_mlp_grad<<<nblk, GT, kSmemGrad, cs>>>(m->P, dx, dt, didx + b0, nb, 1.0f / (float)nb, G, L);
      k_mlp_reduce<<<(NP + 255) / 256, 256, 0, cs>>>(G, L, nblk, m->grad, m->loss, m->acc, (double)nb);
      k_mlp_adam<<<(NP + 255) / 256, 256, 0, cs>>>(m->P, m->M, m->V, m->img, m->grad, lr, b1, b2,
                                                   eps, c1t, c2t, ebase, k);
    }
    ok = ok && cudaStreamEndCapture(cs, &graph) == cudaSuccess &&
         cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
  }
  std::vector<int> perm(n);
  for (int i = 0; i < n; i++) perm[i] = i;
  uint64_t r = seed * 0x9E3779B97F4A7C15ull + 1;
  for (int ep = 0; ep < epochs && ok; ep++) {
    // Fisher-Yates shuffle with a splitmix-style generator
    for (int i = n - 1; i > 0; i--) {
      r += 0x9E3779B97F4A7C15ull;
      uint64_t z = r;
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      z ^= z >> 31;
      const int j = (int)(z % (uint64_t)(i + 1));
      std::swap(perm[i], perm[j]);
    }
    int* order = didx + (cluster && (ep & 1) ? n : 0);
    // the buffer's last reader: two epochs back, or the last one's graph
    if (ep >= (cluster ? 2 : 1)) ok = cudaEventSynchronize(done[cluster ? ep & 1 : 0]) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(order, perm.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, up) == cudaSuccess &&
         cudaStreamSynchronize(up) == cudaSuccess;  // perm is shuffled on
    if (!ok) break;
    if (cluster) {
      EpochArgs A = {m->P, m->M, m->V, m->img, dx, dt, order, n, batch, lr, b1, b2, eps,
                     c1t + (size_t)ep * nbat, c2t + (size_t)ep * nbat, acc + ep};
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at = {};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = nb_per;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.gridDim = dim3(nb_per);
      cfg.blockDim = dim3(GT);
      cfg.dynamicSmemBytes = epoch_smem(nb_per);
      cfg.stream = cs;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      ok = cudaLaunchKernelEx(&cfg, k_mlp_epoch, A) == cudaSuccess &&
           cudaEventRecord(done[ep & 1], cs) == cudaSuccess;
    } else {
      const int eb = ep * nbat;
      ok = cudaMemcpyAsync(ebase, &eb, sizeof(int), cudaMemcpyHostToDevice, cs) == cudaSuccess &&
           cudaMemsetAsync(m->acc, 0, sizeof(double), cs) == cudaSuccess &&
           cudaGraphLaunch(exec, cs) == cudaSuccess &&
           cudaMemcpyAsync(acc + ep, m->acc, sizeof(double), cudaMemcpyDeviceToDevice, cs) == cudaSuccess &&
           cudaEventRecord(done[0], cs) == cudaSuccess;
    }
  }
  if (cs) ok = cudaStreamSynchronize(cs) == cudaSuccess && ok;
  if (ok && losses) {
    std::vector<double> sum(epochs);
    ok = cudaMemcpy(sum.data(), acc, epochs * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess;
    for (int ep = 0; ep < epochs && ok; ep++) losses[ep] = (float)(sum[ep] / n);
  }
  if (ok) m->step += (int)nupd;
  ok = ok && cudaGetLastError() == cudaSuccess;
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  for (auto& e : done)
    if (e) cudaEventDestroy(e);
  if (cs) cudaStreamDestroy(cs);
  if (up) cudaStreamDestroy(up);
  cudaFree(mem);
  return ok ? BL_SUCCESS : BL_FAILURE;
}

}  // extern "C"
