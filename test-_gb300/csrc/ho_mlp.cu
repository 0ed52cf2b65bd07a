// The small network of the learned mode: 48 -> 128 -> 128 -> 128 -> 8,
// GELU (tanh form) after each hidden layer; BF16 operands, FP32 accumulation
// on the tensor cores (mma.sync m16n8k16), FP32 master weights with Adam.
//
//  * train_rows_kernel: the forward and backward passes of training, 32 rows
//    a tile; train_weights_kernel: the weight gradients, split over the rows.
//  * mlp_infer_kernel: the whole forward pass for inference, persistent over
//    128-row tiles, weights resident in shared memory, each warp owning 16
//    rows through all four layers (no block-level synchronisation between
//    layers).
//
// Weight layout: W_l[in][out] row-major (FP32 master and a BF16 copy), plus a
// BF16 transposed copy Wt_l[out][in] for the inference kernel's B operands.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "ho_host.h"
#include "ho_mlp.h"
#include "ho_mlp_infer.cuh"

namespace ho {

// ---------------------------------------------------------------------------
// Training: one forward and backward pass.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// Four 8 x 8 matrices of BF16 from shared memory, each lane giving the address
// of one row (lane l: row l % 8 of matrix l / 8).
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr(p)));
}

constexpr int kTrainRows = 32;             // rows of a tile
constexpr int kHPad = kMlpHidden + 8;      // row strides in shared memory: 16 bytes past a multiple of 128,
constexpr int kXPad = kMlpInPad + 8;       // so that 8 rows of a matrix load hit different banks
struct TrainSmem {
  bf16 w[kMlpInPad + 2 * kMlpHidden][kHPad];  // W_0 (64 rows), W_1, W_2: [in][out]
  bf16 x[kTrainRows][kXPad];
  bf16 h[2][kTrainRows][kHPad];  // activations, then dZ, in turn
  float w3[kMlpHidden][kMlpOut];
  float dy[kTrainRows][kMlpOut];  // the output gradients' BF16 values
  float b[3][kMlpHidden], b3[kMlpOut];
};

// acc += A[16 x K] B[K x 32], A row-major (lda), B either [k][n] (TB false)
// or [n][k] (TB true), both in shared memory with row stride kHPad for B.
template <bool TB>
__device__ __forceinline__ void train_mma(const bf16* A, int lda, const bf16* B, int K, float (&acc)[4][4]) {
  const int l = threadIdx.x & 31;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 16) {
    uint32_t a[4];
    ldsm4(a, A + ((l & 7) + ((l >> 3) & 1) * 8) * lda + k0 + (l >> 4) * 8);
#pragma unroll
    for (int np = 0; np < 2; ++np) {
      uint32_t b[4];
      if (TB) ldsm4(b, B + (np * 16 + (l & 7) + (l >> 4) * 8) * kHPad + k0 + ((l >> 3) & 1) * 8);
      else ldsm4t(b, B + (k0 + (l & 7) + ((l >> 3) & 1) * 8) * kHPad + np * 16 + (l >> 4) * 8);
      mma_bf16(acc[2 * np], a[0], a[1], a[2], a[3], b[0], b[1]);
      mma_bf16(acc[2 * np + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
  }
}

// Columns of the FP32 sums that the rows' pass leaves per block and row half:
// the bias gradients of the four layers, then the loss.
constexpr int kSumCols = 3 * kMlpHidden + kMlpOut + 1;

struct TrainArgs {
  const bf16* w[4];
  const float* b[4];
  float* gb[4];
  bf16* h[4];   // the layers' inputs, rows x (64, 128, 128, 128); h[0] is written only from xf
  bf16* dz[4];  // the gradients before the activations, rows x (128, 128, 128, 8)
  const float* xf;  // FP32 input rows of 48, or nullptr: h[0] holds the BF16 rows
  const float* t;
  const uint8_t* valid;
  float* loss;
  float* sums;  // [2 * row_blocks][kSumCols]
  int row_blocks;
  int rows;
  float inv_n;
};

// Forward and backward for tiles of 32 rows: masked MSE over the first
// kMlpTargets outputs (loss = mean over valid rows of sum_j (y_j - t_j)^2), and
// every layer's gradient before its activation, with the weights in shared
// memory and the activations' slopes in registers (a thread owns the same rows
// and columns of every layer, forward and backward). Eight warps: 2 row halves
// x 4 groups of 32 columns. Bias gradients and the loss are summed from the FP32
// values, a block's part of each kept apart and added up in a fixed order
// (train_weights_kernel), so a call gives the same bits every time.
// What bounds it is the chain of six small products and their barriers; the
// products are 0.6 GFLOP at 4,096 rows. As separate launches per layer (product,
// bias and activation, slope, column sums) the pass ran 28 kernels, 200 us at
// 4,096 rows; this one takes 16 us (19 with its bias gradients by atomics).
__global__ void __launch_bounds__(256) train_rows_kernel(TrainArgs P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3, m0 = 16 * (warp >> 2), n0 = 32 * (warp & 3);
  for (int i = tid; i < (kMlpInPad + 2 * kMlpHidden) * (kMlpHidden / 8); i += 256) {
    const int r = i / (kMlpHidden / 8), v = i % (kMlpHidden / 8);
    const bf16* w = r < kMlpInPad ? P.w[0] + r * kMlpHidden
                                  : (r < kMlpInPad + kMlpHidden ? P.w[1] + (r - kMlpInPad) * kMlpHidden
                                                                : P.w[2] + (r - kMlpInPad - kMlpHidden) * kMlpHidden);
    *reinterpret_cast<uint4*>(&S.w[r][8 * v]) = *reinterpret_cast<const uint4*>(w + 8 * v);
  }
  for (int i = tid; i < kMlpHidden * kMlpOut; i += 256) S.w3[i / kMlpOut][i % kMlpOut] = __bfloat162float(P.w[3][i]);
  for (int i = tid; i < 3 * kMlpHidden; i += 256) S.b[i / kMlpHidden][i % kMlpHidden] = P.b[i / kMlpHidden][i % kMlpHidden];
  if (tid < kMlpOut) S.b3[tid] = P.b[3][tid];
  float sum[3][4][2], sum3 = 0.f, loss = 0.f;
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) sum[l][nt][0] = sum[l][nt][1] = 0.f;
  const int tiles = (P.rows + kTrainRows - 1) / kTrainRows;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = static_cast<int64_t>(tile) * kTrainRows;
    const int live = min(kTrainRows, P.rows - static_cast<int>(row0));
    __syncthreads();  // the weights are in; the tile before is done
    for (int i = tid; i < kTrainRows * (kMlpInPad / 8); i += 256) {
      const int r = i / (kMlpInPad / 8), v = i % (kMlpInPad / 8);
      uint4 q = make_uint4(0u, 0u, 0u, 0u);
      if (r < live) {
        if (P.xf) {
          uint32_t h[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int c = 8 * v + e;
            const uint32_t u = c < kMlpIn ? __float_as_uint(P.xf[(row0 + r) * kMlpIn + c]) : 0u;
            h[e] = (u + 0x7FFFu + ((u >> 16) & 1u)) >> 16;  // round to nearest even
          }
          q = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
          *reinterpret_cast<uint4*>(P.h[0] + (row0 + r) * kMlpInPad + 8 * v) = q;
        } else {
          q = *reinterpret_cast<const uint4*>(P.h[0] + (row0 + r) * kMlpInPad + 8 * v);
        }
      }
      *reinterpret_cast<uint4*>(&S.x[r][8 * v]) = q;
    }
    __syncthreads();
    float acc[4][4], slope[3][4][4];
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      if (l == 0) train_mma<false>(&S.x[m0][0], kXPad, &S.w[0][n0], kMlpInPad, acc);
      else train_mma<false>(&S.h[(l - 1) & 1][m0][0], kHPad, &S.w[l == 1 ? kMlpInPad : kMlpInPad + kMlpHidden][n0],
                            kMlpHidden, acc);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = m0 + g + 8 * h, c = n0 + 8 * nt + 2 * t4;
          const float z0 = acc[nt][2 * h] + S.b[l][c], z1 = acc[nt][2 * h + 1] + S.b[l][c + 1];
          slope[l][nt][2 * h] = gelu_grad(z0);
          slope[l][nt][2 * h + 1] = gelu_grad(z1);
          const __nv_bfloat162 v = __floats2bfloat162_rn(gelu(z0), gelu(z1));
          *reinterpret_cast<__nv_bfloat162*>(&S.h[l & 1][r][c]) = v;
          if (r < live) *reinterpret_cast<__nv_bfloat162*>(P.h[l + 1] + (row0 + r) * kMlpHidden + c) = v;
        }
      __syncthreads();
    }
    {  // output layer and loss: a thread per row and output
      const int r = tid / kMlpOut, j = tid % kMlpOut;
      float y = 0.f;
#pragma unroll 16
      for (int k = 0; k < kMlpHidden; k += 2) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&S.h[0][r][k]));
        y = fmaf(v.x, S.w3[k][j], y);
        y = fmaf(v.y, S.w3[k + 1][j], y);
      }
      float gr = 0.f;
      if (r < live && j < kMlpTargets && P.valid[row0 + r]) {
        const float e = y + S.b3[j] - P.t[(row0 + r) * kMlpOut + j];
        gr = 2.f * e * P.inv_n;
        loss += e * e * P.inv_n;
      }
      sum3 += gr;
      const bf16 gq = __float2bfloat16(gr);
      S.dy[r][j] = __bfloat162float(gq);
      if (r < live) P.dz[3][(row0 + r) * kMlpOut + j] = gq;
    }
    __syncthreads();
#pragma unroll
    for (int l = 2; l >= 0; --l) {
      if (l == 2) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = m0 + g + 8 * (q >> 1), c = n0 + 8 * nt + 2 * t4 + (q & 1);
            float v = 0.f;
#pragma unroll
            for (int o = 0; o < kMlpOut; ++o) v = fmaf(S.dy[r][o], S.w3[c][o], v);
            acc[nt][q] = v;
          }
      } else {
        train_mma<true>(&S.h[(l + 1) & 1][m0][0], kHPad, &S.w[(l == 1 ? kMlpInPad + kMlpHidden : kMlpInPad) + n0][0],
                        kMlpHidden, acc);
      }
      // h[l & 1] was last read before the barrier above
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = m0 + g + 8 * h, c = n0 + 8 * nt + 2 * t4;
          const float v0 = acc[nt][2 * h] * slope[l][nt][2 * h], v1 = acc[nt][2 * h + 1] * slope[l][nt][2 * h + 1];
          sum[l][nt][0] += v0;
          sum[l][nt][1] += v1;
          const __nv_bfloat162 v = __floats2bfloat162_rn(v0, v1);
          if (l > 0) *reinterpret_cast<__nv_bfloat162*>(&S.h[l & 1][r][c]) = v;
          if (r < live) *reinterpret_cast<__nv_bfloat162*>(P.dz[l] + (row0 + r) * kMlpHidden + c) = v;
        }
      if (l > 0) __syncthreads();
    }
  }
  float* sums = P.sums + (2 * static_cast<int64_t>(blockIdx.x) + (warp >> 2)) * kSumCols;
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float v = sum[l][nt][e];
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (g == 0) sums[kMlpHidden * l + n0 + 8 * nt + 2 * t4 + e] = v;
      }
  // the output layer's bias and the loss: the warps' parts through S.dy, which
  // the last tile has read before its last barrier
  float v = sum3;
#pragma unroll
  for (int off = 8; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
  if (lane < kMlpOut) S.dy[warp][lane] = v;
  if (lane == 0) S.dy[8 + warp][0] = loss;
  __syncthreads();
  if ((warp & 3) == 0 && lane <= kMlpOut) {
    float t = 0.f;
    for (int k = 0; k < 4; ++k) t += lane < kMlpOut ? S.dy[warp + k][lane] : S.dy[8 + warp + k][0];
    sums[3 * kMlpHidden + lane] = t;
  }
}

// Weight gradients of all four layers: gW_l += h_l^T dz_l. Block (x, y): output
// tile x of the 12 tiles of 64 x 64 (of 64 x 8 for the output layer) and every
// gridDim.y-th chunk of 256 rows from chunk y on, read whole (16 bytes a load) before
// its products; 8 warps of 16 x 32 outputs. Few output tiles and long sums: the
// split over the rows is what fills the device; below 1,024 rows two parts at
// most, whose sum does not depend on which comes first. Tile 12: the sums that
// the rows' pass left, a warp a column, in a fixed order. (Four launches of one layer
// each, whose operands were read two bytes at a time across rows, took 123 us
// at 4,096 rows; this one takes 10 us, 7 of them without tile 12.)
constexpr int kGradChunk = 256, kGradPad = 72, kGradTiles = 12;
__global__ void __launch_bounds__(256) train_weights_kernel(TrainArgs P, float* __restrict__ g0, float* __restrict__ g1,
                                                            float* __restrict__ g2, float* __restrict__ g3) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* As = reinterpret_cast<bf16*>(smem_raw);
  bf16* Ds = As + kGradChunk * kGradPad;
  const int tile = blockIdx.x;
  if (tile == kGradTiles) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = blockIdx.y * 8 + warp; c < kSumCols; c += 8 * gridDim.y) {
      float v = 0.f;
      for (int k = lane; k < 2 * P.row_blocks; k += 32) v += P.sums[static_cast<int64_t>(k) * kSumCols + c];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0)
        *(c < 3 * kMlpHidden ? P.gb[c / kMlpHidden] + c % kMlpHidden
                             : (c < kSumCols - 1 ? P.gb[3] + c - 3 * kMlpHidden : P.loss)) = v;
    }
    return;
  }
  const int l = tile < 2 ? 0 : (tile < 6 ? 1 : (tile < 10 ? 2 : 3));
  const int q = tile - (l == 0 ? 0 : (l == 1 ? 2 : (l == 2 ? 6 : 10)));
  const int im = l == 0 ? 0 : (l == 3 ? 64 * q : 64 * (q >> 1)), in = l == 3 ? 0 : 64 * (q & 1);
  const int lda = l == 0 ? kMlpInPad : kMlpHidden, ldd = l == 3 ? kMlpOut : kMlpHidden;
  const int rows_in = l == 0 ? kMlpIn : kMlpHidden;
  const int dv = l == 3 ? 1 : 8;  // vectors of 8 in a row of dz that are not padding
  const bf16* A = P.h[l] + im;
  const bf16* D = P.dz[l] + in;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = 16 * (warp >> 1), n0 = 32 * (warp & 1);
  float acc[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  const int chunks = (P.rows + kGradChunk - 1) / kGradChunk;
  for (int ch = blockIdx.y; ch < chunks; ch += gridDim.y) {
    const int64_t row0 = static_cast<int64_t>(ch) * kGradChunk;
    const int live = min(kGradChunk, P.rows - static_cast<int>(row0));
    __syncthreads();
#pragma unroll
    for (int i = tid; i < kGradChunk * 8; i += 256) {
      const int r = i >> 3, v = i & 7;
      uint4 a = make_uint4(0u, 0u, 0u, 0u), e = a;
      if (r < live) {
        a = *reinterpret_cast<const uint4*>(A + (row0 + r) * lda + 8 * v);
        if (v < dv) e = *reinterpret_cast<const uint4*>(D + (row0 + r) * ldd + 8 * v);
      }
      *reinterpret_cast<uint4*>(As + r * kGradPad + 8 * v) = a;
      *reinterpret_cast<uint4*>(Ds + r * kGradPad + 8 * v) = e;
    }
    __syncthreads();
    if (l < 3 || n0 == 0) {
#pragma unroll 4
      for (int k0 = 0; k0 < kGradChunk; k0 += 16) {
        uint32_t a[4];
        ldsm4t(a, As + (k0 + (lane & 7) + (lane >> 4) * 8) * kGradPad + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t b[4];
          ldsm4t(b, Ds + (k0 + (lane & 7) + ((lane >> 3) & 1) * 8) * kGradPad + n0 + np * 16 + (lane >> 4) * 8);
          mma_bf16(acc[2 * np], a[0], a[1], a[2], a[3], b[0], b[1]);
          mma_bf16(acc[2 * np + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
        }
      }
    }
  }
  float* G = l == 0 ? g0 : (l == 1 ? g1 : (l == 2 ? g2 : g3));
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = im + m0 + g + 8 * (e >> 1), n = in + n0 + 8 * nt + 2 * t4 + (e & 1);
      if (m < rows_in && n < ldd) atomicAdd(G + m * ldd + n, acc[nt][e]);
    }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2,
                            bf16* __restrict__ pb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  if (pb) pb[i] = __float2bfloat16(pi);
}

__global__ void gather_rows_kernel(const bf16* __restrict__ X, const float* __restrict__ T,
                                   const uint8_t* __restrict__ V, const int32_t* __restrict__ idx, int B,
                                   bf16* __restrict__ Xb, float* __restrict__ Tb, uint8_t* __restrict__ Vb) {
  const int r = blockIdx.x;
  if (r >= B) return;
  const int64_t s = idx[r];
  for (int c = threadIdx.x; c < kMlpInPad; c += blockDim.x) Xb[static_cast<int64_t>(r) * kMlpInPad + c] = X[s * kMlpInPad + c];
  for (int c = threadIdx.x; c < kMlpOut; c += blockDim.x) Tb[static_cast<int64_t>(r) * kMlpOut + c] = T[s * kMlpOut + c];
  if (threadIdx.x == 0) Vb[r] = V[s];
}

__global__ void transpose_cast_kernel(const float* __restrict__ W, int in, int out, int in_pad, int out_pad,
                                      bf16* __restrict__ Wt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= in_pad * out_pad) return;
  const int o = i / in_pad, k = i % in_pad;
  Wt[i] = __float2bfloat16((o < out && k < in) ? W[k * out + o] : 0.f);
}

// ---------------------------------------------------------------------------
// Fused inference: Y[M x 8] = MLP(X[M x 64]) (X: 48 features + zero pad).
// ---------------------------------------------------------------------------
// Y[M x 8] = MLP(X[M x 64]) (X: 48 features + zero pad); M from m_dev
// (items x rows_per_item) when given.
__global__ void __launch_bounds__(256) mlp_infer_kernel(MlpDev P, const bf16* __restrict__ X, int64_t M,
                                                        const unsigned* __restrict__ m_dev, int rows_per_item,
                                                        float* __restrict__ Y) {
  const int64_t rows = m_dev ? static_cast<int64_t>(*m_dev) * rows_per_item : M;
  mlp_infer_tiles(P, XRows{X}, rows, Y);
}

size_t mlp_infer_smem() { return sizeof(InferSmem); }

int mlp_infer(const MlpDev& P, const void* X, int64_t M, const unsigned* m_dev, int rows_per_item, float* Y,
              cudaStream_t s, int grid) {
  // the attribute is set once per device
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return int(e);
  if (dev < 0 || dev >= 64) return int(cudaErrorInvalidDevice);
  if (!attr[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(InferSmem)));
    if (e != cudaSuccess) return int(e);
    attr[dev].store(true, std::memory_order_release);
  }
  mlp_infer_kernel<<<grid, 256, sizeof(InferSmem), s>>>(P, static_cast<const bf16*>(X), M, m_dev, rows_per_item, Y);
  return int(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Trainer
// ---------------------------------------------------------------------------
static const int kDims[5] = {kMlpInPad, kMlpHidden, kMlpHidden, kMlpHidden, kMlpOut};

#define MLP_TRY(x)                           \
  do {                                       \
    cudaError_t e__ = (x);                   \
    if (e__ != cudaSuccess) return int(e__); \
  } while (0)

int Mlp::alloc() {
  if (ready) return 0;
  for (int l = 0; l < 4; ++l) {
    const int n = kDims[l] * kDims[l + 1];
    MLP_TRY(cudaMalloc(&W[l], n * sizeof(float)));
    MLP_TRY(cudaMalloc(&Wb[l], n * sizeof(bf16)));
    MLP_TRY(cudaMalloc(&mW[l], n * sizeof(float)));
    MLP_TRY(cudaMalloc(&vW[l], n * sizeof(float)));
    MLP_TRY(cudaMalloc(&b[l], kDims[l + 1] * sizeof(float)));
    MLP_TRY(cudaMalloc(&mb[l], kDims[l + 1] * sizeof(float)));
    MLP_TRY(cudaMalloc(&vb[l], kDims[l + 1] * sizeof(float)));
  }
  MLP_TRY(cudaMalloc(&grads, (kMlpParams + 1) * sizeof(float)));
  for (int l = 0, o = 0; l < 4; ++l) {
    gW[l] = grads + o;
    o += (l == 0 ? kMlpIn : kMlpHidden) * kDims[l + 1];
    gb[l] = grads + o;
    o += kDims[l + 1];
  }
  MLP_TRY(cudaMalloc(&wt[0], kMlpHidden * kMlpInPad * sizeof(bf16)));
  MLP_TRY(cudaMalloc(&wt[1], kMlpHidden * kMlpHidden * sizeof(bf16)));
  MLP_TRY(cudaMalloc(&wt[2], kMlpHidden * kMlpHidden * sizeof(bf16)));
  MLP_TRY(cudaMalloc(&wt[3], 16 * kMlpHidden * sizeof(bf16)));
  ready = true;
  return 0;
}

void Mlp::release() {
  for (int l = 0; l < 4; ++l) {
    cudaFree(W[l]); cudaFree(Wb[l]); cudaFree(mW[l]); cudaFree(vW[l]);
    cudaFree(b[l]); cudaFree(mb[l]); cudaFree(vb[l]); cudaFree(wt[l]);
    W[l] = gW[l] = mW[l] = vW[l] = b[l] = gb[l] = mb[l] = vb[l] = nullptr;
    Wb[l] = nullptr;
    wt[l] = nullptr;
  }
  cudaFree(grads);
  grads = nullptr;
  cudaFree(sums);
  sums = nullptr;
  cudaFree(ws);
  ws = nullptr;
  ws_rows = 0;
  ready = false;
  trained = false;
}

// Host-side parameter upload: W_l[in][out] row-major fp32 (in padded to 64
// for layer 0, rows 48..63 must be zero), b_l.
int Mlp::set_params(const float* const* Wh, const float* const* bh, cudaStream_t s) {
  MLP_TRY(cudaError_t(alloc()));
  for (int l = 0; l < 4; ++l) {
    const int n = kDims[l] * kDims[l + 1];
    MLP_TRY(cudaMemcpyAsync(W[l], Wh[l], n * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_TRY(cudaMemcpyAsync(b[l], bh[l], kDims[l + 1] * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_TRY(cudaMemsetAsync(mW[l], 0, n * sizeof(float), s));
    MLP_TRY(cudaMemsetAsync(vW[l], 0, n * sizeof(float), s));
    MLP_TRY(cudaMemsetAsync(mb[l], 0, kDims[l + 1] * sizeof(float), s));
    MLP_TRY(cudaMemsetAsync(vb[l], 0, kDims[l + 1] * sizeof(float), s));
  }
  step = 0;
  return refresh_copies(s);
}

int Mlp::get_params(float* const* Wh, float* const* bh, cudaStream_t s) {
  for (int l = 0; l < 4; ++l) {
    const int n = kDims[l] * kDims[l + 1];
    MLP_TRY(cudaMemcpyAsync(Wh[l], W[l], n * sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_TRY(cudaMemcpyAsync(bh[l], b[l], kDims[l + 1] * sizeof(float), cudaMemcpyDeviceToHost, s));
  }
  return int(cudaStreamSynchronize(s));
}

__global__ void cast_kernel(const float* __restrict__ a, int n, bf16* __restrict__ o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) o[i] = __float2bfloat16(a[i]);
}

int Mlp::refresh_copies(cudaStream_t s) {
  for (int l = 0; l < 4; ++l) {
    const int n = kDims[l] * kDims[l + 1];
    cast_kernel<<<(n + 255) / 256, 256, 0, s>>>(W[l], n, static_cast<bf16*>(Wb[l]));
  }
  transpose_cast_kernel<<<(kMlpHidden * kMlpInPad + 255) / 256, 256, 0, s>>>(W[0], kMlpInPad, kMlpHidden, kMlpInPad,
                                                                            kMlpHidden, static_cast<bf16*>(wt[0]));
  transpose_cast_kernel<<<(kMlpHidden * kMlpHidden + 255) / 256, 256, 0, s>>>(W[1], kMlpHidden, kMlpHidden,
                                                                             kMlpHidden, kMlpHidden, static_cast<bf16*>(wt[1]));
  transpose_cast_kernel<<<(kMlpHidden * kMlpHidden + 255) / 256, 256, 0, s>>>(W[2], kMlpHidden, kMlpHidden,
                                                                             kMlpHidden, kMlpHidden, static_cast<bf16*>(wt[2]));
  transpose_cast_kernel<<<(16 * kMlpHidden + 255) / 256, 256, 0, s>>>(W[3], kMlpHidden, kMlpOut, kMlpHidden, 16,
                                                                      static_cast<bf16*>(wt[3]));
  return int(cudaGetLastError());
}

MlpDev Mlp::dev() const {
  MlpDev d;
  d.w1t = wt[0];
  d.w2t = wt[1];
  d.w3t = wt[2];
  d.w4t = wt[3];
  d.b1 = b[0];
  d.b2 = b[1];
  d.b3 = b[2];
  d.b4 = b[3];
  return d;
}

int Mlp::ensure_ws(int rows) {
  if (rows <= ws_rows) return 0;
  cudaFree(ws);
  ws = nullptr;
  ws_rows = 0;
  // X (64 wide), H1..H3 and dZ0..dZ2 (128 wide), dY (8 wide), in BF16
  MLP_TRY(cudaMalloc(&ws, static_cast<size_t>(rows) * (kMlpInPad + 6 * kMlpHidden + kMlpOut) * sizeof(bf16)));
  ws_rows = rows;
  return 0;
}

// Forward + backward on a batch: rows either Xf (FP32, 48 wide) or Xb (BF16,
// padded to 64). Gradients and, after them, the batch loss overwrite grads.
int Mlp::forward_backward(int B, const float* Xf, const void* Xb, const float* Tb, const uint8_t* Vb, int n_valid,
                          cudaStream_t s) {
  // the shared-memory sizes are set once per device
  static std::atomic<bool> attr[64];
  constexpr int kGradSmem = 2 * kGradChunk * kGradPad * static_cast<int>(sizeof(bf16));
  int dev = 0, sms = 0;
  MLP_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return int(cudaErrorInvalidDevice);
  if (!attr[dev].load(std::memory_order_acquire)) {
    MLP_TRY(cudaFuncSetAttribute(train_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(TrainSmem))));
    MLP_TRY(cudaFuncSetAttribute(train_weights_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
    attr[dev].store(true, std::memory_order_release);
  }
  MLP_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MLP_TRY(cudaError_t(ensure_ws(B)));
  if (!sums) {
    MLP_TRY(cudaMalloc(&sums, static_cast<size_t>(2) * sms * kSumCols * sizeof(float)));
    sums_blocks = sms;
  }
  TrainArgs P;
  bf16* f = static_cast<bf16*>(ws);
  P.h[0] = Xf ? f : static_cast<bf16*>(const_cast<void*>(Xb));
  f += static_cast<size_t>(B) * kMlpInPad;
  for (int l = 1; l < 4; ++l, f += static_cast<size_t>(B) * kMlpHidden) P.h[l] = f;
  for (int l = 0; l < 3; ++l, f += static_cast<size_t>(B) * kMlpHidden) P.dz[l] = f;
  P.dz[3] = f;
  for (int l = 0; l < 4; ++l) {
    P.w[l] = static_cast<const bf16*>(Wb[l]);
    P.b[l] = b[l];
    P.gb[l] = gb[l];
  }
  P.xf = Xf;
  P.t = Tb;
  P.valid = Vb;
  P.loss = grads + kMlpParams;
  P.rows = B;
  P.inv_n = 1.0f / std::max(1, n_valid);
  MLP_TRY(cudaMemsetAsync(grads, 0, (kMlpParams + 1) * sizeof(float), s));
  const int tiles = (B + kTrainRows - 1) / kTrainRows, chunks = (B + kGradChunk - 1) / kGradChunk;
  P.sums = sums;
  P.row_blocks = std::min(tiles, sums_blocks);
  train_rows_kernel<<<P.row_blocks, 256, sizeof(TrainSmem), s>>>(P);
  MLP_TRY(cudaGetLastError());
  train_weights_kernel<<<dim3(kGradTiles + 1, std::min(chunks, B < 1024 ? 2 : 32)), 256, kGradSmem, s>>>(
      P, gW[0], gW[1], gW[2], gW[3]);
  return int(cudaGetLastError());
}

int Mlp::adam_step(float lr, cudaStream_t s) {
  ++step;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - std::pow(b1, static_cast<float>(step)), c2 = 1.f - std::pow(b2, static_cast<float>(step));
  for (int l = 0; l < 4; ++l) {
    const int n = (l == 0 ? kMlpIn : kMlpHidden) * kDims[l + 1];  // layer 0's padding rows stay zero
    adam_kernel<<<(n + 255) / 256, 256, 0, s>>>(W[l], gW[l], mW[l], vW[l], n, lr, b1, b2, eps, c1, c2,
                                                static_cast<bf16*>(Wb[l]));
    adam_kernel<<<(kDims[l + 1] + 255) / 256, 256, 0, s>>>(b[l], gb[l], mb[l], vb[l], kDims[l + 1], lr, b1, b2, eps,
                                                            c1, c2, nullptr);
  }
  return int(cudaGetLastError());
}

int Mlp::train(const void* X, const float* T, const uint8_t* V, int64_t n, int steps, int batch, float lr, uint64_t seed,
               std::vector<float>& losses, cudaStream_t s) {
  bf16* Xb;
  float* Tb;
  uint8_t* Vb;
  int32_t* idx;
  MLP_TRY(cudaMalloc(&Xb, static_cast<size_t>(batch) * kMlpInPad * sizeof(bf16)));
  MLP_TRY(cudaMalloc(&Tb, static_cast<size_t>(batch) * kMlpOut * sizeof(float)));
  MLP_TRY(cudaMalloc(&Vb, batch));
  MLP_TRY(cudaMalloc(&idx, batch * sizeof(int32_t)));
  std::vector<int32_t> hidx(batch);
  Pcg64 rng(seed, 7);
  losses.clear();
  float* hloss = nullptr;
  MLP_TRY(cudaMallocHost(&hloss, sizeof(float) * std::max(1, steps)));
  for (int it = 0; it < steps; ++it) {
    for (int i = 0; i < batch; ++i) hidx[i] = static_cast<int32_t>(rng.next() % static_cast<uint64_t>(n));
    MLP_TRY(cudaMemcpyAsync(idx, hidx.data(), batch * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    gather_rows_kernel<<<batch, 64, 0, s>>>(static_cast<const bf16*>(X), T, V, idx, batch, Xb, Tb, Vb);
    // cosine decay to 5% of lr
    const float lr_t = lr * (0.05f + 0.95f * 0.5f * (1.f + std::cos(3.14159265f * it / std::max(1, steps))));
    int rc = forward_backward(batch, nullptr, Xb, Tb, Vb, batch, s);
    if (rc) return rc;
    rc = adam_step(lr_t, s);
    if (rc) return rc;
    MLP_TRY(cudaMemcpyAsync(hloss + it, grads + kMlpParams, sizeof(float), cudaMemcpyDeviceToHost, s));
    // host copy of the loss waits for the stream only at the end
  }
  MLP_TRY(cudaStreamSynchronize(s));
  losses.assign(hloss, hloss + steps);
  cudaFreeHost(hloss);
  cudaFree(Xb);
  cudaFree(Tb);
  cudaFree(Vb);
  cudaFree(idx);
  const int rc = refresh_copies(s);
  if (rc) return rc;
  trained = true;
  return 0;
}

}  // namespace ho
