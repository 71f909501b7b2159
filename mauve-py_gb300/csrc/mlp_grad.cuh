// Backward pass of the band-proposal MLP, and its forward layers off the TMA
// path (included by mlp.cu after the GELU helpers).  The backward pass is four
// kinds of launch:
//
//   k_grad_top    loss, dO and the 256 -> 2 output layer's gradients, and
//                 dZ3 = (dO W4) * gelu'(Z3)
//   k_grad_z      dZ(l) = (dZ(l+1) W(l+1)) * gelu'(Z(l)), for layers 2 and 1
//   k_grad_w      dW(l) = dZ(l)^T H(l-1) of all three layers, split over rows
//   k_grad_sum    the sums over row splits
//
// dZ is rounded to bf16 for the products (fp32 accumulation); the bias
// gradients are column sums of the fp32 values, taken where they are
// produced.  Every sum over rows is a fixed tree: partial sums per CTA in
// `part`, added up in order by k_grad_sum.
//
// The pass is short of blocks, not of bandwidth or tensor rate, at the
// training batch (4,096 rows: 3.8 GFLOP, 20 MB): one CTA per 64 x 64 tile of
// dW over all rows, loading element by element, took 0.5 ms per layer of the
// pass's 2.1 ms.  Splitting rows so that there are about four CTAs per SM,
// 16-byte asynchronous loads and ldmatrix with transposition (both operands
// of dW are k-strided) bring the pass to 65 us.
#pragma once
#include <cuda_bf16.h>

#include "mvg_common.cuh"

namespace mvg {

constexpr int kGradThreads = 128;
constexpr int kGradTile = 64;             // output tile, both ways
constexpr int kGradK = 32;                // K step
constexpr int kGradPitch = kGradTile + 8;  // shared row pitch of a k-strided tile: 144 bytes, 16-byte aligned, no
                                           // two rows of an 8 x 8 matrix in one bank
constexpr int kGradSplits = 16;            // most row splits of dW
constexpr int kGradSplitRows = 256;        // fewest rows of a split worth its partial tile
constexpr int kGradParts = 128;            // most CTA rows (partial column sums) of k_grad_z
constexpr int kGradTopParts = 512;         // and of k_grad_top

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// A hidden layer of the forward pass for operands off TMA's rules: z = A W^T +
// b, h = GELU(z) for A [M x K], W [256 x K] (K a multiple of 8), a CTA per 64 x
// 64 tile, three stages of 32 columns in flight.  The products are added in the
// order of the plain GEMM it stands in for (k_gemm_bf16, 16 at a time), so its
// results are the same bits; with that and a launch for bias and GELU the forward
// call took 148 us over 1,003 rows and 1.10 ms over 100,001, now 70 and 382.  wide: A may be loaded 16 bytes at a
// time.  z may be null.
__global__ void __launch_bounds__(kGradThreads) k_mlp_layer_mma(const __nv_bfloat16* __restrict__ A, int wide,
                                                                const __nv_bfloat16* __restrict__ W,
                                                                const float* __restrict__ bias, int64_t M, int K,
                                                                float* __restrict__ z, __nv_bfloat16* __restrict__ h) {
  constexpr int kStages = 3, kPitch = kGradK + 8;
  __shared__ __align__(16) __nv_bfloat16 s_a[kStages][kGradTile][kPitch], s_b[kStages][kGradTile][kPitch];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n0 = ((int)blockIdx.x & 3) * kGradTile;
  const int64_t m0 = (int64_t)(blockIdx.x >> 2) * kGradTile;
  const int steps = (K + kGradK - 1) / kGradK, wm = (wid >> 1) * 32, wn = (wid & 1) * 32;
  auto load = [&](int step) {
    const int s = step % kStages;
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(&s_a[s][0][0]);
    const uint32_t b0 = (uint32_t)__cvta_generic_to_shared(&s_b[s][0][0]);
#pragma unroll
    for (int e = tid; e < kGradTile * (kGradK / 8); e += kGradThreads) {
      const int r = e >> 2, q = (e & 3) * 8, k = step * kGradK + q;
      const bool in = k < K, live = in && m0 + r < M;
      cp16(b0 + (r * kPitch + q) * 2, W + (in ? (int64_t)(n0 + r) * K + k : 0), in);
      if (wide) {
        cp16(a0 + (r * kPitch + q) * 2, A + (live ? (m0 + r) * K + k : 0), live);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) s_a[s][r][q + u] = live ? A[(m0 + r) * K + k + u] : __float2bfloat16(0.f);
      }
    }
  };
  float acc[2][4][4] = {};
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) load(s);
    cp_commit();
  }
  for (int step = 0; step < steps; ++step) {
    cp_wait<kStages - 2>();
    __syncthreads();
    if (step + kStages - 1 < steps) load(step + kStages - 1);
    cp_commit();
    const int s = step % kStages;
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(&s_a[s][0][0]);
    const uint32_t b0 = (uint32_t)__cvta_generic_to_shared(&s_b[s][0][0]);
#pragma unroll
    for (int k = 0; k < kGradK; k += 16) {
      uint32_t a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ldsm4(a[i], a0 + ((wm + i * 16 + (lane & 15)) * kPitch + k + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int j = 0; j < 2; ++j)  // matrices (n, k), (n, k + 8), (n + 8, k), (n + 8, k + 8)
        ldsm4(b[j], b0 + ((wn + j * 16 + (lane & 7) + (lane >> 4) * 8) * kPitch + k + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], &b[j >> 1][(j & 1) * 2]);
    }
  }
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int64_t r = m0 + wm + i * 16 + half * 8 + g;
      if (r >= M) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = n0 + wn + j * 8 + 2 * t;
        const float v0 = acc[i][j][2 * half] + bias[c], v1 = acc[i][j][2 * half + 1] + bias[c + 1];
        if (z) *reinterpret_cast<float2*>(z + r * kHid + c) = make_float2(v0, v1);
        *reinterpret_cast<__nv_bfloat162*>(h + r * kHid + c) = __floats2bfloat162_rn(gelu(v0), gelu(v1));
      }
    }
}

// part layout of k_grad_top, per CTA: db3 [256], dW4 [2 x 256], db4 [2], loss.
constexpr int kTopPart = 3 * kHid + 4;

// One column per thread, `rows` rows per CTA.
__global__ void __launch_bounds__(kHid) k_grad_top(const float* __restrict__ o, const float* __restrict__ tgt,
                                                   const __nv_bfloat16* __restrict__ w4,
                                                   const float* __restrict__ z, const __nv_bfloat16* __restrict__ h,
                                                   int64_t n, int64_t rows, __nv_bfloat16* __restrict__ dz,
                                                   float* __restrict__ part) {
  constexpr int kChunk = 32;
  __shared__ float s_d[kChunk][2], s_red[2][3];
  const int col = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * rows, r1 = r0 + rows < n ? r0 + rows : n;
  const float w0 = __bfloat162float(w4[col]), w1 = __bfloat162float(w4[kHid + col]);
  float db = 0.f, dw0 = 0.f, dw1 = 0.f, loss = 0.f, dbo = 0.f;
  for (int64_t c0 = r0; c0 < r1; c0 += kChunk) {
    __syncthreads();
    if (col < 2 * kChunk) {  // thread 2 r + k: output k of the chunk's row r
      const int64_t r = c0 + (col >> 1);
      float g = 0.f;
      if (r < r1) {
        const float diff = o[c0 * kOut + col] - tgt[c0 * kOut + col];
        loss += diff * diff;
        g = 2.f * diff / (float)n;
        dbo += g;
      }
      s_d[col >> 1][col & 1] = __bfloat162float(__float2bfloat16(g));
    }
    __syncthreads();
    const int m = (int)(r1 - c0 < kChunk ? r1 - c0 : kChunk);
#pragma unroll 8
    for (int k = 0; k < m; ++k) {
      const int64_t e = (c0 + k) * kHid + col;
      const float d0 = s_d[k][0], d1 = s_d[k][1], hv = __bfloat162float(h[e]);
      const float v = (d0 * w0 + d1 * w1) * gelu_grad(z[e]);
      dw0 += d0 * hv;
      dw1 += d1 * hv;
      db += v;
      dz[e] = __float2bfloat16(v);
    }
  }
  float* p = part + (int64_t)blockIdx.x * kTopPart;
  p[col] = db;
  p[kHid + col] = dw0;
  p[2 * kHid + col] = dw1;
  if (col < 2 * kChunk) {  // lanes of one parity hold one output
#pragma unroll
    for (int d = 16; d > 1; d >>= 1) {
      dbo += __shfl_xor_sync(0xffffffffu, dbo, d);
      loss += __shfl_xor_sync(0xffffffffu, loss, d);
    }
    loss += __shfl_xor_sync(0xffffffffu, loss, 1);
    if ((col & 31) < 2) s_red[col >> 5][col & 1] = dbo;
    if ((col & 31) == 0) s_red[col >> 5][2] = loss;
  }
  __syncthreads();
  if (col < 3) p[3 * kHid + col] = s_red[0][col] + s_red[1][col];
}

// dz_out = (dz_in W) * gelu'(z) for W [256 x 256], a CTA per 64 columns and
// every gridDim.y-th 64 rows: W's 64 columns stay in shared memory.  Column
// sums of the CTA's rows to part[blockIdx.y].
__global__ void __launch_bounds__(kGradThreads) k_grad_z(const __nv_bfloat16* __restrict__ dz_in,
                                                         const __nv_bfloat16* __restrict__ w,
                                                         const float* __restrict__ z, int64_t n,
                                                         __nv_bfloat16* __restrict__ dz_out,
                                                         float* __restrict__ part) {
  extern __shared__ __align__(16) uint8_t gz_smem[];
  constexpr int kA = kHid + 8;  // row pitch of the row-major dz tile (528 bytes: 16-byte aligned, distinct banks)
  __nv_bfloat16* const ws = reinterpret_cast<__nv_bfloat16*>(gz_smem);  // [256 k][pitch]
  __nv_bfloat16* const as = ws + kHid * kGradPitch;                     // [64 rows][kA]
  __shared__ float s_col[2][kGradTile];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int c0 = blockIdx.x * kGradTile, wm = (wid >> 1) * 32, wn = (wid & 1) * 32;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t ws0 = (uint32_t)__cvta_generic_to_shared(ws), as0 = (uint32_t)__cvta_generic_to_shared(as);
  for (int e = tid; e < kHid * (kGradTile / 8); e += kGradThreads) {
    const int k = e >> 3, q = e & 7;
    cp16(ws0 + (k * kGradPitch + q * 8) * 2, w + (int64_t)k * kHid + c0 + q * 8, true);
  }
  float col[4][2] = {};  // column sums of this thread's eight columns
  for (int64_t m0 = (int64_t)blockIdx.y * kGradTile; m0 < n; m0 += (int64_t)gridDim.y * kGradTile) {
    __syncthreads();
    for (int e = tid; e < kGradTile * (kHid / 8); e += kGradThreads) {
      const int r = e >> 5, q = e & 31;
      const bool live = m0 + r < n;
      cp16(as0 + (r * kA + q * 8) * 2, dz_in + (live ? (m0 + r) * kHid + q * 8 : 0), live);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    float acc[2][4][4] = {};
#pragma unroll 4
    for (int k = 0; k < kHid; k += 16) {
      uint32_t a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ldsm4(a[i], as0 + ((wm + i * 16 + (lane & 15)) * kA + k + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        ldsm4t(b[j], ws0 + ((k + (lane & 15)) * kGradPitch + wn + j * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], &b[j >> 1][(j & 1) * 2]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int64_t r = m0 + wm + i * 16 + half * 8 + g;
        if (r >= n) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t e = r * kHid + c0 + wn + j * 8 + 2 * t;
          const float2 zz = *reinterpret_cast<const float2*>(z + e);
          const float v0 = acc[i][j][2 * half] * gelu_grad(zz.x), v1 = acc[i][j][2 * half + 1] * gelu_grad(zz.y);
          col[j][0] += v0;
          col[j][1] += v1;
          *reinterpret_cast<__nv_bfloat162*>(dz_out + e) = __floats2bfloat162_rn(v0, v1);
        }
      }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float v = col[j][q];
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
      if (g == 0) s_col[wid >> 1][wn + j * 8 + 2 * t + q] = v;
    }
  __syncthreads();
  if (tid < kGradTile) part[(int64_t)blockIdx.y * kHid + c0 + tid] = s_col[0][tid] + s_col[1][tid];
}
constexpr int kGradZSmem = (kHid * kGradPitch + kGradTile * (kHid + 8)) * 2;

struct GradW {  // one layer of k_grad_w: dW [256 x din] = dz^T in
  const __nv_bfloat16* dz;
  const __nv_bfloat16* in;
  float* part;  // [split][256 x din]
  int din;
  int wide;  // 1: `in` may be loaded 16 bytes at a time
  int tile;  // first tile (blockIdx.x) of this layer
};
struct GradWs {
  GradW l[3];
};

// A 64 x 64 tile of one layer's dW over the rows [blockIdx.y * rows, + rows):
// three stages of 32 rows in flight.
__global__ void __launch_bounds__(kGradThreads) k_grad_w(const __grid_constant__ GradWs P, int64_t n, int64_t rows) {
  constexpr int kStages = 3;
  __shared__ __align__(16) __nv_bfloat16 s_a[kStages][kGradK][kGradPitch], s_b[kStages][kGradK][kGradPitch];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int layer = (int)blockIdx.x >= P.l[1].tile ? (int)blockIdx.x >= P.l[2].tile ? 2 : 1 : 0;
  const GradW& L = P.l[layer];
  const int ntn = (L.din + kGradTile - 1) / kGradTile;
  const int m0 = ((int)blockIdx.x - L.tile) / ntn * kGradTile, n0 = ((int)blockIdx.x - L.tile) % ntn * kGradTile;
  const int64_t r0 = (int64_t)blockIdx.y * rows, r1 = r0 + rows < n ? r0 + rows : n;
  const int steps = r1 > r0 ? (int)((r1 - r0 + kGradK - 1) / kGradK) : 0;
  const int wm = (wid >> 1) * 32, wn = (wid & 1) * 32;
  auto load = [&](int step) {
    const int s = step % kStages;
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(&s_a[s][0][0]);
    const uint32_t b0 = (uint32_t)__cvta_generic_to_shared(&s_b[s][0][0]);
#pragma unroll
    for (int e = tid; e < kGradK * 8; e += kGradThreads) {
      const int k = e >> 3, q = (e & 7) * 8;
      const int64_t r = r0 + (int64_t)step * kGradK + k;
      const bool live = r < r1;
      cp16(a0 + (k * kGradPitch + q) * 2, L.dz + (live ? r * kHid + m0 + q : 0), live);
      const bool inside = live && n0 + q < L.din;  // din is a multiple of 8
      if (L.wide) {
        cp16(b0 + (k * kGradPitch + q) * 2, L.in + (inside ? r * L.din + n0 + q : 0), inside);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u)
          s_b[s][k][q + u] = inside ? L.in[r * L.din + n0 + q + u] : __float2bfloat16(0.f);
      }
    }
  };
  float acc[2][4][4] = {};
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) load(s);
    cp_commit();
  }
  for (int step = 0; step < steps; ++step) {
    cp_wait<kStages - 2>();
    __syncthreads();
    if (step + kStages - 1 < steps) load(step + kStages - 1);
    cp_commit();
    const int s = step % kStages;
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(&s_a[s][0][0]);
    const uint32_t b0 = (uint32_t)__cvta_generic_to_shared(&s_b[s][0][0]);
#pragma unroll
    for (int k = 0; k < kGradK; k += 16) {
      uint32_t a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)  // matrices (k, m), (k, m + 8), (k + 8, m), (k + 8, m + 8), transposed
        ldsm4t(a[i], a0 + ((k + (lane & 7) + (lane >> 4) * 8) * kGradPitch + wm + i * 16 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        ldsm4t(b[j], b0 + ((k + (lane & 15)) * kGradPitch + wn + j * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], &b[j >> 1][(j & 1) * 2]);
    }
  }
  float* out = L.part + (int64_t)blockIdx.y * kHid * L.din;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + wn + j * 8 + 2 * t;
      if (c >= L.din) continue;
#pragma unroll
      for (int half = 0; half < 2; ++half)
        *reinterpret_cast<float2*>(out + (int64_t)(m0 + wm + i * 16 + half * 8 + g) * L.din + c) =
            make_float2(acc[i][j][2 * half], acc[i][j][2 * half + 1]);
    }
}

// One stretch of the flat gradient: out[e] = sum over k < parts of
// part[k * pitch + e].
struct GradSeg {
  const float* part;
  float* out;
  int64_t len, pitch;
  int parts;
  float scale;
};
constexpr int kGradSegs = 9;
struct GradSegs {
  GradSeg s[kGradSegs];
  int block[kGradSegs + 1];  // first block of each
};

// 128 outputs per block, the parts over its eight rows of threads.
__global__ void __launch_bounds__(1024) k_grad_sum(const __grid_constant__ GradSegs P) {
  __shared__ float sum[8][128];
  int k = 0;
  while ((int)blockIdx.x >= P.block[k + 1]) ++k;
  const GradSeg& S = P.s[k];
  const int64_t e = (int64_t)((int)blockIdx.x - P.block[k]) * 128 + (threadIdx.x & 127);
  const int row = threadIdx.x >> 7;
  float v = 0.f;
  if (e < S.len)
#pragma unroll 4
    for (int q = row; q < S.parts; q += 8) v += S.part[q * S.pitch + e];
  sum[row][threadIdx.x & 127] = v;
  __syncthreads();
  if (row == 0 && e < S.len) {
    float a = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) a += sum[q][threadIdx.x];
    S.out[e] = a * S.scale;
  }
}

}  // namespace mvg
