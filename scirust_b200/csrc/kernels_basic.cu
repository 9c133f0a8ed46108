// Bandwidth-bound training kernels: RMSNorm fwd/bwd, RoPE fwd/bwd, SwiGLU fwd/bwd,
// embedding gather / deterministic scatter-add, fused softmax-cross-entropy
// (loss + gradient in place), deterministic sum of squares, fused AdamW over a flat
// parameter buffer, casts. bf16 storage, fp32 math, RNE rounding on store.
//
// Semantics follow the reference's scalar CUDA-C kernels
// (scirust-cuda/src/chain.rs: rmsnorm_fast :423, rope :225/:350, swiglu :55/:278,
// embed :247/:579, ce_loss_grad :637, adamw_norm :707, sumsq :742/:759) but the
// shapes are different: 16-byte vector accesses, warp-per-row reductions with a
// fixed shuffle tree (bitwise repeatable, no atomics), one launch per flat buffer.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>
#include "api.h"

#include "dependent.cuh"
#include "rope_rows.cuh"

namespace sb {

__device__ __forceinline__ float bflo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bfhi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t packbf(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  f[0] = bflo(v.x); f[1] = bfhi(v.x); f[2] = bflo(v.y); f[3] = bfhi(v.y);
  f[4] = bflo(v.z); f[5] = bfhi(v.z); f[6] = bflo(v.w); f[7] = bfhi(v.w);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(packbf(f[0], f[1]), packbf(f[2], f[3]), packbf(f[4], f[5]), packbf(f[6], f[7]));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------
// RMSNorm forward: y = x * rsqrt(mean(x^2) + eps) * w. One warp per row.
// Optionally stores inv_rms (fp32 per row) for the backward pass.
// ---------------------------------------------------------------------------
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                   __nv_bfloat16* __restrict__ y, float* __restrict__ inv_rms, int rows, int cols,
                                   int ldx, int ldy, float eps) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const __nv_bfloat16* xr = x + static_cast<size_t>(row) * ldx;
  // eight interleaved accumulators (iteration i of the lane goes to accumulator i % 8), added in
  // index order: more loads in flight, and the same association as the fused prologue of the decode
  // GEMV, which spreads the eight accumulators over eight warps
  float acc[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) acc[a] = 0.f;
  for (int c0 = lane * 8; c0 < cols; c0 += 8 * 256) {
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int c = c0 + a * 256;
      if (c < cols) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(xr + c), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[a] += f[j] * f[j];
      }
    }
  }
  float ss = acc[0];
#pragma unroll
  for (int a = 1; a < 8; ++a) ss += acc[a];
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / static_cast<float>(cols) + eps);
  if (inv_rms && lane == 0) inv_rms[row] = inv;
  __nv_bfloat16* yr = y + static_cast<size_t>(row) * ldy;
  for (int c = lane * 8; c < cols; c += 256) {
    float f[8], g[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + c), f);
    unpack8(*reinterpret_cast<const uint4*>(w + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * inv * g[j];
    *reinterpret_cast<uint4*>(yr + c) = pack8(f);
  }
}

// The same for few rows, one CTA of eight warps per row: with a row per warp a decode batch leaves most SMs idle and each
// row pays its loads one after another. Warp a computes accumulator a of the kernel above and the eight are added in
// index order, so the results are the same bits. 64 rows of 4096: 7.2 us above, 2.3 us here.
__global__ void __launch_bounds__(256)
rmsnorm_fwd_row_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* y, float* inv_rms, int cols,
                       int ldx, int ldy, float eps) {
  pdl_trigger();
  pdl_wait();
  __shared__ float s_acc[8][32];
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __nv_bfloat16* xr = x + static_cast<size_t>(row) * ldx;
  constexpr int KEEP = 4;                       // 16-byte words of the row a thread keeps (rows up to 8192)
  uint4 kept[KEEP], kw[KEEP];
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int c = threadIdx.x * 8 + i * 2048;
    if (c < cols) {
      kept[i] = *reinterpret_cast<const uint4*>(xr + c);
      kw[i] = *reinterpret_cast<const uint4*>(w + c);
    }
  }
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    if (threadIdx.x * 8 + i * 2048 < cols) {
      float f[8];
      unpack8(kept[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += f[j] * f[j];
    }
  }
  for (int c = threadIdx.x * 8 + KEEP * 2048; c < cols; c += 2048) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + c), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += f[j] * f[j];
  }
  s_acc[warp][lane] = acc;
  __syncthreads();
  float ss = s_acc[0][lane];
#pragma unroll
  for (int a = 1; a < 8; ++a) ss += s_acc[a][lane];
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / static_cast<float>(cols) + eps);
  if (inv_rms && threadIdx.x == 0) inv_rms[row] = inv;
  __nv_bfloat16* yr = y + static_cast<size_t>(row) * ldy;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int c = threadIdx.x * 8 + i * 2048;
    if (c < cols) {
      float f[8], g[8];
      unpack8(kept[i], f);
      unpack8(kw[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * inv * g[j];
      *reinterpret_cast<uint4*>(yr + c) = pack8(f);
    }
  }
  for (int c = threadIdx.x * 8 + KEEP * 2048; c < cols; c += 2048) {
    float f[8], g[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + c), f);
    unpack8(*reinterpret_cast<const uint4*>(w + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * inv * g[j];
    *reinterpret_cast<uint4*>(yr + c) = pack8(f);
  }
}

// RMSNorm backward, input gradient. With g = dy*w and r = inv_rms:
//   dx = r * (g - x * r^2 * mean(g*x))   (+ optional residual-stream gradient `dres`)
// Every rounding is spelt out: left to the compiler, which product of a sum it contracts changes with the code around it, and a dx that
// rounds otherwise in a few places moves every gradient below it by its last bits. g = a * w is exact (two bf16 values).
__device__ __forceinline__ float rms_dot(float dot, float a, float g, float b) { return __fmaf_rn(__fmul_rn(a, g), b, dot); }
// Rows that stay in registers (512, 1024 and 2048 columns): r * (g - b k), one rounding in the bracket, and then d.
__device__ __forceinline__ float rms_dx_reg(float r, float k, float a, float g, float b) {
  return __fmul_rn(r, __fmaf_rn(-b, k, __fmul_rn(a, g)));
}
__global__ void rmsnorm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                      const __nv_bfloat16* __restrict__ w, const float* __restrict__ inv_rms,
                                      const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                      int rows, int cols) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t off = static_cast<size_t>(row) * cols;
  float dot = 0.f;
  for (int c = lane * 8; c < cols; c += 256) {
    float a[8], b[8], g[8];
    unpack8(*reinterpret_cast<const uint4*>(dy + off + c), a);
    unpack8(*reinterpret_cast<const uint4*>(x + off + c), b);
    unpack8(*reinterpret_cast<const uint4*>(w + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) dot = rms_dot(dot, a[j], g[j], b[j]);
  }
  dot = warp_sum(dot);
  const float r = inv_rms[row];
  const float k = r * r * dot / static_cast<float>(cols);
  for (int c = lane * 8; c < cols; c += 256) {
    float a[8], b[8], g[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(dy + off + c), a);
    unpack8(*reinterpret_cast<const uint4*>(x + off + c), b);
    unpack8(*reinterpret_cast<const uint4*>(w + c), g);
    // here b k is rounded before it is subtracted, and d is added in the rounding of the product
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = __fmaf_rn(a[j], g[j], -__fmul_rn(b[j], k));
    if (dres) {
      float d[8];
      unpack8(*reinterpret_cast<const uint4*>(dres + off + c), d);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = __fmaf_rn(r, o[j], d[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = __fmul_rn(r, o[j]);
    }
    *reinterpret_cast<uint4*>(dx + off + c) = pack8(o);
  }
}

// The same for rows of NV * 256 columns (NV <= 8): dy and x of the row stay in registers, all loads are issued
// before the first use, and the sum runs in the order of the general kernel.
template <int NV>
__global__ void rmsnorm_bwd_dx_reg_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                          const __nv_bfloat16* __restrict__ w, const float* __restrict__ inv_rms,
                                          const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                          int rows) {
  constexpr int cols = NV * 256;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t off = static_cast<size_t>(row) * cols;
  uint4 va[NV], vb[NV], vg[NV], vd[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane * 8 + i * 256;
    va[i] = *reinterpret_cast<const uint4*>(dy + off + c);
    vb[i] = *reinterpret_cast<const uint4*>(x + off + c);
    vg[i] = *reinterpret_cast<const uint4*>(w + c);
    if (dres) vd[i] = *reinterpret_cast<const uint4*>(dres + off + c);
  }
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float a[8], b[8], g[8];
    unpack8(va[i], a); unpack8(vb[i], b); unpack8(vg[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) dot = rms_dot(dot, a[j], g[j], b[j]);
  }
  dot = warp_sum(dot);
  const float r = inv_rms[row];
  const float k = r * r * dot / static_cast<float>(cols);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float a[8], b[8], g[8], o[8];
    unpack8(va[i], a); unpack8(vb[i], b); unpack8(vg[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = rms_dx_reg(r, k, a[j], g[j], b[j]);
    if (dres) {
      float d[8];
      unpack8(vd[i], d);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = __fadd_rn(o[j], d[j]);
    }
    *reinterpret_cast<uint4*>(dx + off + lane * 8 + i * 256) = pack8(o);
  }
}

// RMSNorm gain gradient, stage 1: partial[ry][j] = sum over the rows of chunk ry of
// dy*x*inv_rms, rows visited in ascending order by each warp, warps combined in warp
// order. Stage 2 (colsum_finish_kernel) adds the chunks in chunk order.
__global__ void rmsnorm_bwd_dw_partial_kernel(const __nv_bfloat16* __restrict__ dy,
                                              const __nv_bfloat16* __restrict__ x,
                                              const float* __restrict__ inv_rms, float* __restrict__ partial,
                                              int rows, int cols, int rows_per_chunk) {
  __shared__ float red[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 256 + lane * 8;
  const int r0 = blockIdx.y * rows_per_chunk;
  const int r1 = min(rows, r0 + rows_per_chunk);
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < cols) {
    // four rows of this warp in flight; the adds keep the row order
    for (int r = r0 + warp; r < r1; r += 32) {
      uint4 va[4], vb[4];
      float iv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int rr = r + 8 * u;
        if (rr < r1) {
          va[u] = *reinterpret_cast<const uint4*>(dy + static_cast<size_t>(rr) * cols + c);
          vb[u] = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(rr) * cols + c);
          iv[u] = inv_rms[rr];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r + 8 * u < r1) {
          float a[8], b[8];
          unpack8(va[u], a);
          unpack8(vb[u], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] += a[j] * b[j] * iv[u];
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int t = threadIdx.x;
  float s = 0.f;
#pragma unroll
  for (int wdx = 0; wdx < 8; ++wdx) s += red[wdx][t];
  const int col = blockIdx.x * 256 + t;
  if (col < cols) partial[static_cast<size_t>(blockIdx.y) * cols + col] = s;
}


// Both gradients in one pass, for rows of NV * 256 columns (NV <= 4 by its registers; 512 and 1024 are the widths that the models here
// have, 256 and 768 keep two passes and have not been timed): dy and x are read once and not twice. A warp takes every
// (warps of the grid)-th row, keeps the row in registers as above (the same dx to the bit) and adds its share of the gain's gradient to NV * 8
// sums per lane; the warps of a CTA are added in warp order, the CTAs in stage 2. Two CTAs of eight warps per SM: 128 registers
// hold the row and the sums, the gain lies in shared memory (with one CTA per SM this form lost to two passes). Bound by memory: 16384 x 1024
// with a residual 21.4 + 14.4 + 4.3 us in two passes and their stage 2, 26.7 + 4.4 so; 999 x 1024 3.3 + 7.1 + 1.9 / 4.3 + 2.7.
constexpr int RB_WARPS = 8;
template <int NV, bool RES>
__global__ void __launch_bounds__(RB_WARPS * 32, 2)
rmsnorm_bwd_both_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                        const __nv_bfloat16* __restrict__ w, const float* __restrict__ inv_rms,
                        const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int rows) {
  constexpr int cols = NV * 256;
  __shared__ float red[RB_WARPS][cols];
  __shared__ uint4 s_w[cols / 8];                        // the gain: in registers it would cost spills
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  }
  if (threadIdx.x < cols / 8) s_w[threadIdx.x] = *reinterpret_cast<const uint4*>(w + threadIdx.x * 8);
  __syncthreads();
  for (int row = blockIdx.x * RB_WARPS + warp; row < rows; row += gridDim.x * RB_WARPS) {
    const size_t off = static_cast<size_t>(row) * cols + lane * 8;
    uint4 va[NV], vb[NV], vd[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      va[i] = *reinterpret_cast<const uint4*>(dy + off + i * 256);
      vb[i] = *reinterpret_cast<const uint4*>(x + off + i * 256);
      if (RES) vd[i] = *reinterpret_cast<const uint4*>(dres + off + i * 256);
    }
    const float r = inv_rms[row];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float a[8], b[8], g[8];
      unpack8(va[i], a); unpack8(vb[i], b); unpack8(s_w[lane + i * 32], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        dot = rms_dot(dot, a[j], g[j], b[j]);
        acc[i][j] += a[j] * b[j] * r;
      }
    }
    dot = warp_sum(dot);
    // the words are unpacked again below: kept as 64 floats across the sum they would spill
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      asm volatile("" : "+r"(va[i].x), "+r"(va[i].y), "+r"(va[i].z), "+r"(va[i].w));
      asm volatile("" : "+r"(vb[i].x), "+r"(vb[i].y), "+r"(vb[i].z), "+r"(vb[i].w));
    }
    const float k = r * r * dot / static_cast<float>(cols);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float a[8], b[8], g[8], o[8];
      unpack8(va[i], a); unpack8(vb[i], b); unpack8(s_w[lane + i * 32], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rms_dx_reg(r, k, a[j], g[j], b[j]);
      if (RES) {
        float d[8];
        unpack8(vd[i], d);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __fadd_rn(o[j], d[j]);
      }
      *reinterpret_cast<uint4*>(dx + off + i * 256) = pack8(o);
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    *reinterpret_cast<float4*>(&red[warp][lane * 8 + i * 256]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float4*>(&red[warp][lane * 8 + i * 256 + 4]) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += RB_WARPS * 32) {
    float s = red[0][c];
#pragma unroll
    for (int v = 1; v < RB_WARPS; ++v) s += red[v][c];
    partial[static_cast<size_t>(blockIdx.x) * cols + c] = s;
  }
}

// Stage 2 for many partial rows: 32 columns per CTA, 32 lanes of partials each (lane l adds l, l + 32, ... in order), lanes added in
// order. A thread of colsum_finish_kernel walks all partials of its column: 64 x 1024 4.3 us, 296 x 1024 here 4.4.
__global__ void __launch_bounds__(1024)
colsum_finish_lanes_kernel(const float* __restrict__ partial, int parts, int cols, float* __restrict__ out_f32,
                           __nv_bfloat16* __restrict__ out_bf16) {
  __shared__ float s[32][33];
  const int c = threadIdx.x & 31, l = threadIdx.x >> 5, col = blockIdx.x * 32 + c;
  float v = 0.f;
  if (col < cols) {
#pragma unroll 10
    for (int k = l; k < parts; k += 32) v += __ldg(partial + static_cast<size_t>(k) * cols + col);
  }
  s[l][c] = v;
  __syncthreads();
  if (l || col >= cols) return;
#pragma unroll
  for (int k = 1; k < 32; ++k) v += s[k][c];
  if (out_f32) out_f32[col] = v;
  if (out_bf16) out_bf16[col] = __float2bfloat16_rn(v);
}

// Generic fixed-order column sum finish: out[j] = sum_k partial[k][j] (k ascending);
// writes fp32 and/or bf16.
__global__ void colsum_finish_kernel(const float* __restrict__ partial, int chunks, int cols,
                                     float* __restrict__ out_f32, __nv_bfloat16* __restrict__ out_bf16) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cols) return;
  float s = 0.f;
  for (int k = 0; k < chunks; ++k) s += partial[static_cast<size_t>(k) * cols + j];
  if (out_f32) out_f32[j] = s;
  if (out_bf16) out_bf16[j] = __float2bfloat16_rn(s);
}

// ---------------------------------------------------------------------------
// SwiGLU over a fused [gate | up] activation: gu is [rows, 2*ff], h is [rows, ff].
// ---------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* h, int rows, int ff) {
  pdl_trigger();
  pdl_wait();
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int per_row = ff >> 3;
  if (idx >= static_cast<size_t>(rows) * per_row) return;
  const size_t r = idx / per_row;
  const int c = static_cast<int>(idx - r * per_row) * 8;
  float g[8], u[8], o[8];
  unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * ff + c), g);
  unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * ff + ff + c), u);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  *reinterpret_cast<uint4*>(h + r * ff + c) = pack8(o);
}

// dgu = [dh*u*silu'(g) | dh*silu(g)], silu'(g) = s*(1 + g*(1-s)), s = sigmoid(g).
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dh,
                                  __nv_bfloat16* __restrict__ dgu, int rows, int ff) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int per_row = ff >> 3;
  if (idx >= static_cast<size_t>(rows) * per_row) return;
  const size_t r = idx / per_row;
  const int c = static_cast<int>(idx - r * per_row) * 8;
  float g[8], u[8], d[8], dg[8], du[8];
  unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * ff + c), g);
  unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * ff + ff + c), u);
  unpack8(*reinterpret_cast<const uint4*>(dh + r * ff + c), d);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float s = 1.f / (1.f + __expf(-g[j]));
    dg[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
    du[j] = d[j] * g[j] * s;
  }
  *reinterpret_cast<uint4*>(dgu + r * 2 * ff + c) = pack8(dg);
  *reinterpret_cast<uint4*>(dgu + r * 2 * ff + ff + c) = pack8(du);
}

// out = a + b (bf16), 8 elements per thread.
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ out, size_t n8) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  float x[8], y[8];
  unpack8(reinterpret_cast<const uint4*>(a)[i], x);
  unpack8(reinterpret_cast<const uint4*>(b)[i], y);
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] += y[j];
  reinterpret_cast<uint4*>(out)[i] = pack8(x);
}

// ---------------------------------------------------------------------------
// Embedding gather (out row i = table row tokens[i]; ids clamped to the table) and
// its deterministic backward: tokens are sorted (stable) on the device beforehand;
// one block per sorted position, only segment heads do work and add their segment's
// rows in sorted order into the table gradient (which may already hold the tied
// LM-head weight gradient).
// ---------------------------------------------------------------------------
__global__ void embed_fwd_kernel(const __nv_bfloat16* __restrict__ table, const int64_t* __restrict__ tokens,
                                 __nv_bfloat16* __restrict__ out, int n, int d, int vocab) {
  const int i = blockIdx.x;
  if (i >= n) return;
  int64_t t = tokens[i];
  if (t < 0) t = 0;
  if (t >= vocab) t = vocab - 1;
  const uint4* src = reinterpret_cast<const uint4*>(table + static_cast<size_t>(t) * d);
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(i) * d);
  for (int c = threadIdx.x; c < (d >> 3); c += blockDim.x) dst[c] = src[c];
}

// The embedding's gradient: rows of dy added to the table's row of their token, in fp32 and in the order of their positions.
constexpr int EB_THREADS = 128, EB_SHORT = 32, EB_SCAN = 8;
__device__ __forceinline__ int eb_token(int64_t t, int vocab) {
  return t < 0 ? 0 : t >= vocab ? vocab - 1 : static_cast<int>(t);
}
// A thread's columns: eight from c + w * EB_STEP, w < W, of a row; a CTA takes EB_THREADS * W words of 16 bytes of it.
constexpr int EB_STEP = EB_THREADS * 8;
__device__ __forceinline__ void eb_add(const uint4& v, float (&to)[8]) {
  float f[8];
  unpack8(v, f);
#pragma unroll
  for (int k = 0; k < 8; ++k) to[k] += f[k];
}
// Rows at(0) .. at(m - 1) one after the other, the words of R rows on their way at once. The whole warp comes here.
template <int W, int R, class At>
__device__ __forceinline__ void eb_add_rows(const __nv_bfloat16* col, const At& at, int m, int c, int d, float (&acc)[W][8]) {
  for (int j0 = 0; j0 < m; j0 += R) {
    uint4 v[R][W];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const size_t row = static_cast<size_t>(at(j0 + u)) * d;
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (j0 + u < m && c + w * EB_STEP < d) v[u][w] = __ldg(reinterpret_cast<const uint4*>(col + row + w * EB_STEP));
    }
#pragma unroll
    for (int u = 0; u < R; ++u)
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (j0 + u < m && c + w * EB_STEP < d) eb_add(v[u][w], acc[w]);
  }
}

// From sorted tokens (stable, so the positions of a token ascend), in two launches. Runs of up to EB_SHORT places: a CTA per place looks
// whether it heads one and adds its rows, one load of a thread at a time in 32 registers, so that all threads of an SM have one; where tokens
// are spread this is what counts (131072 of 128256, d 1024: 133 us, with four rows in flight and fewer CTAs 220).
__global__ void __launch_bounds__(EB_THREADS, 2048 / EB_THREADS)
embed_bwd_short_runs_kernel(const __nv_bfloat16* __restrict__ dy, const int64_t* __restrict__ sorted_tok, const int64_t* __restrict__ perm,
                            __nv_bfloat16* __restrict__ dtable, int n, int d, int vocab, int accumulate) {
  const int i = blockIdx.x;
  const int64_t here = sorted_tok[i], before = sorted_tok[max(i - 1, 0)], far = sorted_tok[min(i + EB_SHORT, n - 1)];
  const int t = eb_token(here, vocab);
  if ((i > 0 && eb_token(before, vocab) == t) || (i + EB_SHORT < n && eb_token(far, vocab) == t)) return;
  for (int c = threadIdx.x; c < (d >> 3); c += EB_THREADS) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint4* dst = reinterpret_cast<uint4*>(dtable + static_cast<size_t>(t) * d) + c;
    if (accumulate) unpack8(*dst, acc);
    for (int j = i; j < n && eb_token(sorted_tok[j], vocab) == t; ++j)
      eb_add(reinterpret_cast<const uint4*>(dy + static_cast<size_t>(perm[j]) * d)[c], acc);
    *dst = pack8(acc);
  }
}
// Longer runs, whose rows are one chain of additions: eight on their way at once. A run of more than EB_SHORT places holds a place that is a
// multiple of EB_SHORT; the CTA of the first of these takes it. Each warp reads the places by itself, 32 at a time and the next 32 while
// the rows of these come, and passes positions by shuffles. 65536 tokens of 32000 with frequencies 1 / rank, d 1024: 3735 us one row at a
// time, 956 so, d 4096 from 131072 29170 / 2108.
static_assert(EB_SHORT == 32, "a warp looks back over the places before its own");
__global__ void __launch_bounds__(EB_THREADS)
embed_bwd_long_runs_kernel(const __nv_bfloat16* __restrict__ dy, const int64_t* __restrict__ sorted_tok, const int64_t* __restrict__ perm,
                           __nv_bfloat16* __restrict__ dtable, int n, int d, int vocab, int accumulate) {
  const int place = blockIdx.x * EB_SHORT, lane = threadIdx.x & 31, c = (blockIdx.y * EB_THREADS + threadIdx.x) * 8;
  if (c - lane * 8 >= d) return;                          // no column for this warp
  const int t = eb_token(sorted_tok[place], vocab);
  const int back = place - 1 - lane;
  const uint32_t same = __ballot_sync(0xffffffffu, back >= 0 && eb_token(sorted_tok[back], vocab) == t);
  if (same == 0xffffffffu) return;                        // the place EB_SHORT before is of the run too
  const int first = place - __popc(same);
  if (first + EB_SHORT >= n || eb_token(sorted_tok[first + EB_SHORT], vocab) != t) return;
  uint4* dst = reinterpret_cast<uint4*>(dtable + static_cast<size_t>(t) * d + c);
  float acc[1][8] = {};
  if (accumulate && c < d) unpack8(*dst, acc[0]);
  auto read = [&](int p) { return p < n && eb_token(sorted_tok[p], vocab) == t ? static_cast<int>(perm[p]) : -1; };
  int mine = read(first + lane);
  for (int base = first + 32;; base += 32) {
    const int m = __popc(__ballot_sync(0xffffffffu, mine >= 0));        // a run is in one piece
    const int next = m == 32 ? read(base + lane) : -1;
    eb_add_rows<1, 8>(dy + c, [&](int j) { return __shfl_sync(0xffffffffu, mine, j & 31); }, m, c, d, acc);
    if (m < 32) break;
    mine = next;
  }
  if (c < d) *dst = pack8(acc[0]);
}

// From the tokens as they are, without sorting them: three launches (a memset among them) instead of a radix sort's
// ten. The positions of a token are chained through `next` from `head` by atomic exchanges, in whatever order those happen; a CTA
// per position (and 1024, 2048 or 4096 columns, as the rows are long) looks whether its position heads the chain, puts the chain's positions in ascending order and adds
// their rows in that order, so the sums do not depend on the chain's. Up to EB_SHORT positions are ranked in a warp; a longer
// chain (padding, spaces) is not followed: the CTA reads the tokens from the front, 1024 at a time, and keeps those that are its own,
// which is why the tokens may not be too many (ops/basic.py).
// Bound by the rows of dy and of the table. 16384 tokens of 32000, d 1024: 110 us with the sort before it, 20 so.
__global__ void __launch_bounds__(256)
embed_chain_kernel(const int64_t* __restrict__ tokens, int* __restrict__ head, int* __restrict__ next, int n, int vocab) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) next[i] = atomicExch(head + eb_token(tokens[i], vocab), i);
}
template <int W>
__global__ void __launch_bounds__(EB_THREADS)
embed_bwd_chain_kernel(const __nv_bfloat16* __restrict__ dy, const int64_t* __restrict__ tokens, const int* __restrict__ head,
                       const int* __restrict__ next, __nv_bfloat16* __restrict__ dtable, int n, int d, int vocab, int accumulate) {
  __shared__ int s_list[EB_THREADS * EB_SCAN];
  __shared__ int s_count[EB_SCAN * (EB_THREADS / 32)];
  __shared__ int s_n;
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = (blockIdx.y * (EB_THREADS * W) + threadIdx.x) * 8;
  const int t = eb_token(tokens[i], vocab);
  // all that a token of a single position needs is asked for before the first answer is used
  const int first = head[t], after = next[i];
  __nv_bfloat16* dst = dtable + static_cast<size_t>(t) * d + c;
  const __nv_bfloat16* col = dy + c;
  uint4 own[W], old[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    own[w] = old[w] = make_uint4(0u, 0u, 0u, 0u);
    if (c + w * EB_STEP < d) {
      own[w] = __ldg(reinterpret_cast<const uint4*>(col + static_cast<size_t>(i) * d + w * EB_STEP));
      if (accumulate && first == i) old[w] = *reinterpret_cast<const uint4*>(dst + w * EB_STEP);
    }
  }
  if (first != i) return;                                // the same for the whole CTA
  float acc[W][8];
#pragma unroll
  for (int w = 0; w < W; ++w) unpack8(old[w], acc[w]);
  auto add_rows = [&](int m) { eb_add_rows<W, 4 / W>(col, [&](int j) { return s_list[min(j, m - 1)]; }, m, c, d, acc); };
  if (after < 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) eb_add(own[w], acc[w]);
  } else {
    if (warp == 0) {
      int m = 0, at = i, mine = 0x7fffffff;              // the whole warp follows the chain; lane j keeps its j-th position
      while (at >= 0 && m < EB_SHORT) {
        if (lane == m) mine = at;
        at = next[at];
        ++m;
      }
      int rank = 0;
#pragma unroll
      for (int j = 0; j < EB_SHORT; ++j) rank += __shfl_sync(0xffffffffu, mine, j) < mine ? 1 : 0;
      if (lane < m) s_list[rank] = mine;
      if (lane == 0) s_n = at >= 0 ? -1 : m;
    }
    __syncthreads();
    const int m = s_n;
    if (m >= 0) {
      add_rows(m);
    } else {
      for (int base = 0; base < n; base += EB_THREADS * EB_SCAN) {
        __syncthreads();                                 // the list of the round before has been read
        uint32_t hit = 0;
        int64_t tk[EB_SCAN];
#pragma unroll
        for (int u = 0; u < EB_SCAN; ++u) {
          const int p = base + u * EB_THREADS + threadIdx.x;
          tk[u] = p < n ? __ldg(tokens + p) : 0;
        }
#pragma unroll
        for (int u = 0; u < EB_SCAN; ++u) {
          const int p = base + u * EB_THREADS + threadIdx.x;
          const bool is = p < n && eb_token(tk[u], vocab) == t;
          const uint32_t b = __ballot_sync(0xffffffffu, is);
          if (is) hit |= 1u << u;
          if (lane == 0) s_count[u * (EB_THREADS / 32) + warp] = __popc(b);
          tk[u] = __popc(b & ((1u << lane) - 1));        // hits of lower lanes
        }
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int u = 0; u < EB_SCAN; ++u) {
#pragma unroll
          for (int w = 0; w < EB_THREADS / 32; ++w) {
            if (w == warp) before = total;
            total += s_count[u * (EB_THREADS / 32) + w];
          }
          if (hit >> u & 1u) s_list[before + static_cast<int>(tk[u])] = base + u * EB_THREADS + threadIdx.x;
        }
        __syncthreads();
        add_rows(total);
      }
    }
  }
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (c + w * EB_STEP < d) *reinterpret_cast<uint4*>(dst + w * EB_STEP) = pack8(acc[w]);
}

// ---------------------------------------------------------------------------
// Fused softmax cross-entropy. One block per row: pass 1 online (max, sum) with a
// fixed combine tree, pass 2 writes d = (softmax - onehot) * grad_scale over the
// logits in place (or to `dlogits`). Target ids >= cols clamp to cols-1; rows whose
// target is negative contribute zero loss and zero gradient (ignore index).
// ---------------------------------------------------------------------------
struct MaxSum { float m, s; };
__device__ __forceinline__ MaxSum ms_combine(MaxSum a, MaxSum b) {
  const float m = fmaxf(a.m, b.m);
  MaxSum r;
  r.m = m;
  r.s = a.s * __expf(a.m - m) + b.s * __expf(b.m - m);
  return r;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS)
ce_fwd_bwd_kernel(const __nv_bfloat16* logits, const int64_t* __restrict__ targets,   // dlogits may be logits
                  float* __restrict__ loss_rows, __nv_bfloat16* dlogits, int rows, int cols, int ld,
                  float grad_scale) {
  __shared__ MaxSum red[THREADS / 32];
  const int r = blockIdx.x;
  if (r >= rows) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const __nv_bfloat16* lr = logits + static_cast<size_t>(r) * ld;
  int64_t tgt = targets[r];
  const bool ignore = tgt < 0;
  if (tgt >= cols) tgt = cols - 1;
  // read before the barrier below: past it other threads may already overwrite the row with its gradient
  const float x_tgt = ignore ? 0.f : __bfloat162float(lr[tgt]);
  MaxSum acc;
  acc.m = -FLT_MAX;                 // below every finite logit: a row of the type's lowest value still has a maximum
  acc.s = 0.f;
  for (int c = tid * 8; c < cols; c += THREADS * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(lr + c), f);
    float mx = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, f[j]);
    const float m = fmaxf(acc.m, mx);
    float s = acc.s * __expf(acc.m - m);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
    acc.m = m;
    acc.s = s;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum other;
    other.m = __shfl_xor_sync(0xffffffffu, acc.m, o);
    other.s = __shfl_xor_sync(0xffffffffu, acc.s, o);
    // combine in a lane-symmetric way so every lane holds identical bits
    acc = (lane & o) ? ms_combine(other, acc) : ms_combine(acc, other);
  }
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  MaxSum tot = red[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) tot = ms_combine(tot, red[w]);
  if (tid == 0) loss_rows[r] = ignore ? 0.f : -(x_tgt - tot.m) + logf(tot.s);
  if (!dlogits) return;
  __nv_bfloat16* dr = dlogits + static_cast<size_t>(r) * ld;
  if (ignore) {
    for (int c = tid * 8; c < cols; c += THREADS * 8) *reinterpret_cast<uint4*>(dr + c) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const float inv = 1.f / tot.s;
  for (int c = tid * 8; c < cols; c += THREADS * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(lr + c), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(f[j] - tot.m) * inv;
      if (c + j == tgt) p -= 1.f;
      f[j] = p * grad_scale;
    }
    *reinterpret_cast<uint4*>(dr + c) = pack8(f);
  }
}

// Rows of up to 512 * 8 * CE_KEEP columns: the row is read once and stays in registers, where the kernel above reads it a
// second time for the gradient (it remains for longer rows). Bound by the bytes of the logits (a read and a write) and,
// close behind, by two exponentials and about ten instructions per element; 64 KB of loads in flight per CTA, two
// CTAs per SM. The maximum is taken first, in packed bf16, so the sum needs no rescaling. It is subtracted before the
// product with log2(e), in packed pairs, so that the error depends on the distance from the maximum and not on the size of
// the logits. 16384 x 32000: 502 us above, 332 us here (6.3 TB/s).
constexpr int CE_THREADS = 512, CE_KEEP = 8;
__device__ __forceinline__ float ce_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// f = exp(f - m) for eight values, m given as -m
__device__ __forceinline__ void ce_exp8(float (&f)[8], float neg_m) {
  constexpr float LOG2E = 1.4426950408889634f;
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    asm("{ .reg .b64 x, y;\n"
        "mov.b64 x, {%0, %1}; mov.b64 y, {%2, %2}; add.rn.f32x2 x, x, y;\n"
        "mov.b64 y, {%3, %3}; mul.rn.f32x2 x, x, y; mov.b64 {%0, %1}, x; }"
        : "+f"(f[j]), "+f"(f[j + 1]) : "f"(neg_m), "f"(LOG2E));
    f[j] = ce_ex2(f[j]);
    f[j + 1] = ce_ex2(f[j + 1]);
  }
}
__global__ void __launch_bounds__(CE_THREADS, 2)
ce_fwd_bwd_row_kernel(const __nv_bfloat16* logits, const int64_t* __restrict__ targets,   // dlogits may be logits
                      float* __restrict__ loss_rows, __nv_bfloat16* dlogits, int cols, int ld,
                      float grad_scale) {
  __shared__ float red_m[CE_THREADS / 32], red_s[CE_THREADS / 32];
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const __nv_bfloat16* lr = logits + static_cast<size_t>(r) * ld;
  constexpr uint32_t NEG2 = 0xff80ff80u;                            // two bf16 infinities, negative
  uint4 v[CE_KEEP];
#pragma unroll
  for (int i = 0; i < CE_KEEP; ++i) {
    const int c = (tid + i * CE_THREADS) * 8;
    v[i] = c < cols ? __ldcs(reinterpret_cast<const uint4*>(lr + c)) : make_uint4(NEG2, NEG2, NEG2, NEG2);
  }
  int64_t tgt = targets[r];
  const bool ignore = tgt < 0;
  if (tgt >= cols) tgt = cols - 1;
  const float x_tgt = ignore ? 0.f : __bfloat162float(lr[tgt]);   // before the row is overwritten (the barriers below)
  uint32_t m2 = NEG2;
  auto widen = [&](uint32_t w) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&m2), b = *reinterpret_cast<const __nv_bfloat162*>(&w);
    const __nv_bfloat162 h = __hmax2(a, b);
    m2 = *reinterpret_cast<const uint32_t*>(&h);
  };
#pragma unroll
  for (int i = 0; i < CE_KEEP; ++i) { widen(v[i].x); widen(v[i].y); widen(v[i].z); widen(v[i].w); }
  float m = fmaxf(fmaxf(__uint_as_float(m2 << 16), __uint_as_float(m2 & 0xffff0000u)), -FLT_MAX);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red_m[warp] = m;
  __syncthreads();
  m = red_m[0];
#pragma unroll
  for (int w = 1; w < CE_THREADS / 32; ++w) m = fmaxf(m, red_m[w]);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < CE_KEEP; ++i) {
    if ((tid + i * CE_THREADS) * 8 < cols) {
      float f[8];
      unpack8(v[i], f);
      ce_exp8(f, -m);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += f[j];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red_s[warp] = s;
  __syncthreads();
  s = red_s[0];
#pragma unroll
  for (int w = 1; w < CE_THREADS / 32; ++w) s += red_s[w];
  if (tid == 0) loss_rows[r] = ignore ? 0.f : -(x_tgt - m) + logf(s);
  if (!dlogits) return;
  __nv_bfloat16* dr = dlogits + static_cast<size_t>(r) * ld;
  if (ignore) {
    for (int c = tid * 8; c < cols; c += CE_THREADS * 8) *reinterpret_cast<uint4*>(dr + c) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const float k = grad_scale / s;
#pragma unroll
  for (int i = 0; i < CE_KEEP; ++i) {
    const int c = (tid + i * CE_THREADS) * 8;
    if (c < cols) {
      float f[8];
      unpack8(v[i], f);
      ce_exp8(f, -m);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] *= k;
      if (static_cast<uint64_t>(tgt - c) < 8u) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c + j == tgt) f[j] -= grad_scale;
      }
      *reinterpret_cast<uint4*>(dr + c) = pack8(f);
    }
  }
}

// ---------------------------------------------------------------------------
// Vocabulary-parallel softmax cross-entropy: every rank holds the logits of its vocabulary shard
// [v0, v0 + cols). Phase 1 writes per-row (max, sum exp(x - max), target logit or 0) of the shard;
// the ranks combine the three numbers; phase 2 turns the shard's logits into
// (exp(x - lse) - onehot) * grad_scale with the global log-sum-exp. Rows with a negative target
// contribute nothing.
// ---------------------------------------------------------------------------
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
ce_shard_stats_kernel(const __nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets,
                      float* __restrict__ stats, int rows, int cols, int ld, int v0) {
  __shared__ MaxSum red[THREADS / 32];
  const int r = blockIdx.x;
  if (r >= rows) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const __nv_bfloat16* lr = logits + static_cast<size_t>(r) * ld;
  MaxSum acc;
  acc.m = -3.0e38f;
  acc.s = 0.f;
  for (int c = tid * 8; c < cols; c += THREADS * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(lr + c), f);
    float mx = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, f[j]);
    const float m = fmaxf(acc.m, mx);
    float s = acc.s * __expf(acc.m - m);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
    acc.m = m;
    acc.s = s;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum other;
    other.m = __shfl_xor_sync(0xffffffffu, acc.m, o);
    other.s = __shfl_xor_sync(0xffffffffu, acc.s, o);
    acc = (lane & o) ? ms_combine(other, acc) : ms_combine(acc, other);
  }
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (tid == 0) {
    MaxSum tot = red[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) tot = ms_combine(tot, red[w]);
    const int64_t tgt = targets[r] - v0;
    stats[r * 3 + 0] = tot.m;
    stats[r * 3 + 1] = tot.s;
    stats[r * 3 + 2] = (tgt >= 0 && tgt < cols && targets[r] >= 0) ? __bfloat162float(lr[tgt]) : 0.f;
  }
}

__global__ void __launch_bounds__(512)
ce_shard_grad_kernel(const __nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets,
                     const float* __restrict__ lse, __nv_bfloat16* __restrict__ dlogits, int rows, int cols, int ld,
                     int v0, float grad_scale) {
  const int r = blockIdx.x;
  if (r >= rows) return;
  const __nv_bfloat16* lr = logits + static_cast<size_t>(r) * ld;
  __nv_bfloat16* dr = dlogits + static_cast<size_t>(r) * ld;
  const bool ignore = targets[r] < 0;
  const int64_t tgt = targets[r] - v0;
  const float l = lse[r];
  const float gs = ignore ? 0.f : grad_scale;
  for (int c = threadIdx.x * 8; c < cols; c += 512 * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(lr + c), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(f[j] - l);
      if (c + j == tgt) p -= 1.f;
      f[j] = p * gs;
    }
    *reinterpret_cast<uint4*>(dr + c) = pack8(f);
  }
}

// ---------------------------------------------------------------------------
// Deterministic sum of squares of a flat bf16 or fp32 buffer: one fp32 partial per
// block (fixed tree), then a single block adds the partials in a fixed strided order.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float ld_as_float(const T* p, size_t i);
template <>
__device__ __forceinline__ float ld_as_float<__nv_bfloat16>(const __nv_bfloat16* p, size_t i) {
  return __bfloat162float(p[i]);
}
template <>
__device__ __forceinline__ float ld_as_float<float>(const float* p, size_t i) { return p[i]; }

// Elements summed by one block of sumsq_partial_kernel (= one partial): 256 threads x 16 strided reads.
// sb_sumsq and sb_sumsq_no_alloc both size their launch from this one constant.
constexpr size_t kSumsqElemsPerPartial = 4096;

template <typename T>
__global__ void sumsq_partial_kernel(const T* __restrict__ g, size_t n, float* __restrict__ partials) {
  __shared__ float red[8];
  float v = 0.f;
  const size_t base = static_cast<size_t>(blockIdx.x) * kSumsqElemsPerPartial;
#pragma unroll 4
  for (int k = 0; k < static_cast<int>(kSumsqElemsPerPartial / 256); ++k) {
    const size_t i = base + k * 256 + threadIdx.x;
    if (i < n) {
      const float x = ld_as_float<T>(g, i);
      v += x * x;
    }
  }
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[w];
    partials[blockIdx.x] = s;
  }
}
// The same partials with one warp per 4096 elements and 16-byte loads, eight of them in flight per lane: bound by the
// bytes of the gradient, where the block above spends a launch slot, a barrier and 2-byte loads on 8 KB. Needs a
// 16-byte aligned buffer. 60 M bf16 elements: 43.8 us above, 26.1 here (4.6 TB/s); the last, partial 4096 by words too (4095
// bf16 elements: 5.2 us one by one, 4.2 so).
template <typename T>
__global__ void __launch_bounds__(256)
sumsq_partial_vec_kernel(const T* __restrict__ g, size_t n, unsigned n_partials, float* __restrict__ partials) {
  const unsigned w = blockIdx.x * 8u + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= n_partials) return;
  const size_t base = static_cast<size_t>(w) * kSumsqElemsPerPartial;
  const bool whole = base + kSumsqElemsPerPartial <= n;
  constexpr int PER = 16 / sizeof(T);                    // elements per word
  const int words = whole ? static_cast<int>(kSumsqElemsPerPartial) / PER : static_cast<int>(n - base) / PER;
  const uint4* g4 = reinterpret_cast<const uint4*>(g + base);
  float a[4] = {0.f, 0.f, 0.f, 0.f};
  auto add = [&](const uint4 (&x)[8]) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if constexpr (sizeof(T) == 2) {
        float f[8];
        unpack8(x[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j & 3] += f[j] * f[j];
      } else {
        const float f[4] = {__uint_as_float(x[u].x), __uint_as_float(x[u].y), __uint_as_float(x[u].z), __uint_as_float(x[u].w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] += f[j] * f[j];
      }
    }
  };
  if (whole) {
    for (int k0 = lane; k0 < static_cast<int>(kSumsqElemsPerPartial) / PER; k0 += 256) {
      uint4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __ldg(g4 + k0 + u * 32);
      add(x);
    }
  } else {
    for (int k0 = lane; k0 < words; k0 += 256) {
      uint4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = k0 + u * 32 < words ? __ldg(g4 + k0 + u * 32) : make_uint4(0u, 0u, 0u, 0u);
      add(x);
    }
  }
  float v = (a[0] + a[1]) + (a[2] + a[3]);
  const size_t last = base + static_cast<size_t>(words) * PER + lane;   // elements behind the last whole word
  if (!whole && last < n) {
    const float x = ld_as_float<T>(g, last);
    v += x * x;
  }
  v = warp_sum(v);
  if (lane == 0) partials[w] = v;
}
__global__ void sumsq_finish_kernel(const float* partials, int n_partials, float* out, int accumulate) {
  __shared__ float red[32];
  pdl_trigger();
  pdl_wait();
  float v = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < n_partials; i += 1024) v += partials[i];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 32; ++w) s += red[w];
    out[0] = accumulate ? out[0] + s : s;
  }
}

// ---------------------------------------------------------------------------
// Fused AdamW / Adam / SGD-momentum over a flat parameter buffer.
// fp32 master p, fp32 m/v, gradient bf16 or fp32, fresh bf16 copy of p written for the
// next forward. The clip factor is derived on the device from grad_sumsq[0]
// (sum of squares of the whole model's gradient): non-finite => the update is
// skipped, norm > max_grad_norm => gradients are scaled by max/norm. Elements at
// index >= decay_end (norm gains, biases) take no weight decay.
// mode: 0 = AdamW (decoupled decay), 1 = Adam (L2 decay folded into g), 2 = SGD
// with momentum (m is the velocity, v unused).
// ---------------------------------------------------------------------------
// One element of the update; shared by the scalar and the 4-wide kernels so both give the same bits.
__device__ __forceinline__ void optim_update_one(float& pi, float& mi, float& vi, float g, float wdi, float lr,
                                                 float b1, float b2, float eps, float bc1, float bc2, int mode) {
  if (mode == 2) {
    if (wdi > 0.f) g += wdi * pi;
    const float vel = b1 * mi + g;
    mi = vel;
    pi -= lr * vel;
  } else {
    if (mode == 1 && wdi > 0.f) g += wdi * pi;
    mi = b1 * mi + (1.f - b1) * g;
    vi = b2 * vi + (1.f - b2) * g * g;
    const float mhat = mi / bc1;
    const float vhat = vi / bc2;
    if (mode == 0) pi -= lr * (mhat / (sqrtf(vhat) + eps) + wdi * pi);
    else pi -= lr * mhat / (sqrtf(vhat) + eps);
  }
}

__device__ __forceinline__ bool optim_clip_scale(const float* grad_sumsq, float max_grad_norm, float grad_scale,
                                                 float& scale) {
  scale = grad_scale;
  if (grad_sumsq) {
    const float sq = grad_sumsq[0] * grad_scale * grad_scale;
    const float norm = sqrtf(sq);
    if (!(sq >= 0.f) || sq > 3.0e38f) return false;  // NaN / inf gradient: skip the whole update
    if (max_grad_norm > 0.f && norm > max_grad_norm) scale *= max_grad_norm / norm;
  }
  return true;
}

template <typename G>
__global__ void optim_step_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                                  const G* __restrict__ grad, __nv_bfloat16* __restrict__ p_bf16, size_t first,
                                  size_t n, size_t decay_end, float lr, float b1, float b2, float eps, float wd,
                                  float bc1, float bc2, const float* __restrict__ grad_sumsq, float max_grad_norm,
                                  float grad_scale, int mode) {
  const size_t i = first + static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float scale;
  if (!optim_clip_scale(grad_sumsq, max_grad_norm, grad_scale, scale)) return;
  const float g = ld_as_float<G>(grad, i) * scale;
  float pi = p[i], mi = m[i], vi = (mode == 2) ? 0.f : v[i];
  optim_update_one(pi, mi, vi, g, (i < decay_end) ? wd : 0.f, lr, b1, b2, eps, bc1, bc2, mode);
  m[i] = mi;
  if (mode != 2) v[i] = vi;
  p[i] = pi;
  if (p_bf16) p_bf16[i] = __float2bfloat16_rn(pi);
}

// Four elements per thread with 16-byte accesses (the update streams 28 bytes per parameter, so it is
// bound by memory bandwidth); covers [0, n4 * 4), 16-byte aligned buffers. The gradient's norm has just been taken from front
// to back, so what is left of the gradient in L2 is its end: blocks walk from the back, and p, m and v, which are used once, pass
// through L2 first to be evicted. 60 M parameters, bf16 gradient, behind the norm: 256 us, 248 so (before / now with the norm:
// 293 / 279).
template <typename G>
__global__ void optim_step_vec4_kernel(float* p, float* m, float* v, const G* grad, __nv_bfloat16* p_bf16, size_t n4,
                                       size_t decay_end, float lr, float b1, float b2, float eps, float wd,
                                       float bc1, float bc2, const float* grad_sumsq,
                                       float max_grad_norm, float grad_scale, int mode) {
  pdl_wait();
  const size_t t = static_cast<size_t>(gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n4) return;
  const size_t i = t * 4;
  float4 pv = __ldcs(reinterpret_cast<const float4*>(p + i));
  float4 mv = __ldcs(reinterpret_cast<const float4*>(m + i));
  float4 vv = (mode == 2) ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcs(reinterpret_cast<const float4*>(v + i));
  float g[4];
  if constexpr (sizeof(G) == 2) {
    const uint2 raw = *reinterpret_cast<const uint2*>(grad + i);
    g[0] = __uint_as_float(raw.x << 16); g[1] = __uint_as_float(raw.x & 0xffff0000u);
    g[2] = __uint_as_float(raw.y << 16); g[3] = __uint_as_float(raw.y & 0xffff0000u);
  } else {
    const float4 raw = *reinterpret_cast<const float4*>(grad + i);
    g[0] = raw.x; g[1] = raw.y; g[2] = raw.z; g[3] = raw.w;
  }
  float scale;
  if (!optim_clip_scale(grad_sumsq, max_grad_norm, grad_scale, scale)) return;
  float* pp = &pv.x; float* mm = &mv.x; float* vp = &vv.x;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    optim_update_one(pp[j], mm[j], vp[j], g[j] * scale, (i + j < decay_end) ? wd : 0.f, lr, b1, b2, eps, bc1, bc2, mode);
  __stcs(reinterpret_cast<float4*>(m + i), mv);
  if (mode != 2) __stcs(reinterpret_cast<float4*>(v + i), vv);
  __stcs(reinterpret_cast<float4*>(p + i), pv);
  if (p_bf16) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(pv.x, pv.y), hi = __floats2bfloat162_rn(pv.z, pv.w);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&lo);
    o.y = *reinterpret_cast<uint32_t*>(&hi);
    __stcs(reinterpret_cast<uint2*>(p_bf16 + i), o);
  }
}

__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, size_t n,
                                        float scale) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(in[i] * scale);
}
__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, size_t n,
                                        float scale) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __bfloat162float(in[i]) * scale;
}

}  // namespace sb

using namespace sb;
#define STREAM static_cast<cudaStream_t>(stream)
#define CHECK_LAUNCH() return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH
static inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// A CTA per row while all of them fit the GPU at once (eight of 256 threads on each SM) and the rows are long enough to give
// most of its threads a word: us, a row per warp against a CTA per row, 1184 rows of 2816 4.6 / 3.8, 512 of 1024 2.5 / 2.1,
// 296 of 256 1.94 / 1.85, but 768 of 1024 2.6 / 2.8, 1184 of 2048 3.5 / 3.6, 1024 of 256 2.1 / 3.0.
static inline bool rms_few_rows(int rows, int cols) { return rows <= 296 || (rows <= 1184 && 2 * rows <= cols); }
extern "C" int sb_rmsnorm_fwd(const void* x, const void* w, void* y, float* inv_rms, int rows, int cols, int ldx,
                              int ldy, float eps, void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 7) || (ldx & 7) || (ldy & 7)) return SB_ERR_ARG;
  if (!al16(x) || !al16(w) || !al16(y)) return SB_ERR_ALIGN;
  if (rms_few_rows(rows, cols)) {
    return launch_dep(rmsnorm_fwd_row_kernel, dim3(rows), dim3(256), 0, STREAM, static_cast<const __nv_bfloat16*>(x),
                      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y), inv_rms, cols, ldx, ldy,
                      eps) == cudaSuccess ? 0 : SB_ERR_LAUNCH;
  }
  const int wpb = 4;
  rmsnorm_fwd_kernel<<<(rows + wpb - 1) / wpb, wpb * 32, 0, STREAM>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y),
      inv_rms, rows, cols, ldx, ldy, eps);
  CHECK_LAUNCH();
}

// The two gradients in one pass: 512 or 1024 columns, partial of parts * cols floats. `parts` CTAs, at most one per eight rows: the order
// of the gain gradient's sum follows from (rows, cols, parts).
extern "C" int sb_rmsnorm_bwd_both(const void* dy, const void* x, const void* w, const float* inv_rms, const void* dres, void* dx,
                                   float* partial, int parts, float* dw_f32, void* dw_bf16, int rows, int cols, void* stream) {
  if (rows <= 0 || parts <= 0 || !partial || (cols != 512 && cols != 1024)) return SB_ERR_ARG;
  if (!al16(dy) || !al16(x) || !al16(w) || !al16(dx) || (dres && !al16(dres))) return SB_ERR_ALIGN;
  const int need = (rows + RB_WARPS - 1) / RB_WARPS;
  if (parts > need) parts = need;
  auto kern = cols == 1024 ? (dres ? rmsnorm_bwd_both_kernel<4, true> : rmsnorm_bwd_both_kernel<4, false>)
                           : (dres ? rmsnorm_bwd_both_kernel<2, true> : rmsnorm_bwd_both_kernel<2, false>);
  kern<<<parts, RB_WARPS * 32, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),
                                            static_cast<const __nv_bfloat16*>(w), inv_rms, static_cast<const __nv_bfloat16*>(dres),
                                            static_cast<__nv_bfloat16*>(dx), partial, rows);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  colsum_finish_lanes_kernel<<<(cols + 31) / 32, 1024, 0, STREAM>>>(partial, parts, cols, dw_f32, static_cast<__nv_bfloat16*>(dw_bf16));
  CHECK_LAUNCH();
}

// dw_partial: fp32 workspace of ceil(rows/rows_per_chunk)*cols floats; rows_per_chunk
// is fixed at 256 so the summation tree depends only on (rows, cols).
extern "C" int sb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* inv_rms, const void* dres,
                              void* dx, float* dw_partial, float* dw_f32, void* dw_bf16, int rows, int cols,
                              void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 7)) return SB_ERR_ARG;
  if (!al16(dy) || !al16(x) || !al16(w) || !al16(dx) || (dres && !al16(dres))) return SB_ERR_ALIGN;
  const int wpb = 4;
  const dim3 dgrid((rows + wpb - 1) / wpb);
  const __nv_bfloat16 *pdy = static_cast<const __nv_bfloat16*>(dy), *px = static_cast<const __nv_bfloat16*>(x),
                      *pw = static_cast<const __nv_bfloat16*>(w), *pres = static_cast<const __nv_bfloat16*>(dres);
  __nv_bfloat16* pdx = static_cast<__nv_bfloat16*>(dx);
  if (cols == 1024) rmsnorm_bwd_dx_reg_kernel<4><<<dgrid, wpb * 32, 0, STREAM>>>(pdy, px, pw, inv_rms, pres, pdx, rows);
  else if (cols == 2048) rmsnorm_bwd_dx_reg_kernel<8><<<dgrid, wpb * 32, 0, STREAM>>>(pdy, px, pw, inv_rms, pres, pdx, rows);
  else if (cols == 512) rmsnorm_bwd_dx_reg_kernel<2><<<dgrid, wpb * 32, 0, STREAM>>>(pdy, px, pw, inv_rms, pres, pdx, rows);
  else rmsnorm_bwd_dx_kernel<<<dgrid, wpb * 32, 0, STREAM>>>(pdy, px, pw, inv_rms, pres, pdx, rows, cols);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  if (dw_partial) {
    const int rpc = 256;
    const int chunks = (rows + rpc - 1) / rpc;
    dim3 grid((cols + 255) / 256, chunks);
    rmsnorm_bwd_dw_partial_kernel<<<grid, 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dy),
                                                            static_cast<const __nv_bfloat16*>(x), inv_rms,
                                                            dw_partial, rows, cols, rpc);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
    colsum_finish_kernel<<<(cols + 255) / 256, 256, 0, STREAM>>>(dw_partial, chunks, cols, dw_f32,
                                                                 static_cast<__nv_bfloat16*>(dw_bf16));
  }
  CHECK_LAUNCH();
}

extern "C" int sb_rope(void* x, int ld, int rows, int n_heads, int dh, int seq_len, int offset,
                       const int* positions, const float* cos_t, const float* sin_t, int backward, void* stream) {
  if (rows <= 0 || n_heads <= 0 || (dh & 7) || (ld & 7) || seq_len <= 0) return SB_ERR_ARG;
  if (!al16(x) || !al16(cos_t) || !al16(sin_t)) return SB_ERR_ALIGN;
  RopeRows p = {};
  p.x = static_cast<__nv_bfloat16*>(x);
  p.ld = ld; p.rows = rows; p.rot_heads = p.heads = n_heads; p.dh = dh;
  p.seq_len = seq_len; p.offset = offset; p.positions = positions;
  p.cos_t = cos_t; p.sin_t = sin_t; p.sign = backward ? -1.f : 1.f;
  return launch_rope_rows<false>(p, STREAM) == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_swiglu_fwd(const void* gu, void* h, int rows, int ff, void* stream) {
  if (rows <= 0 || (ff & 7) || !al16(gu) || !al16(h)) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(rows) * (ff >> 3);
  return launch_dep(swiglu_fwd_kernel, dim3(static_cast<unsigned>((total + 255) / 256)), dim3(256), 0, STREAM,
                    static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(h), rows, ff) == cudaSuccess
             ? 0 : SB_ERR_LAUNCH;
}
extern "C" int sb_swiglu_bwd(const void* gu, const void* dh, void* dgu, int rows, int ff, void* stream) {
  if (rows <= 0 || (ff & 7) || !al16(gu) || !al16(dh) || !al16(dgu)) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(rows) * (ff >> 3);
  swiglu_bwd_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, STREAM>>>(
      static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dh),
      static_cast<__nv_bfloat16*>(dgu), rows, ff);
  CHECK_LAUNCH();
}
extern "C" int sb_add_bf16(const void* a, const void* b, void* out, size_t n, void* stream) {
  if ((n & 7) || !al16(a) || !al16(b) || !al16(out)) return SB_ERR_ARG;
  const size_t n8 = n >> 3;
  add_bf16_kernel<<<static_cast<unsigned>((n8 + 255) / 256), 256, 0, STREAM>>>(
      static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b), static_cast<__nv_bfloat16*>(out),
      n8);
  CHECK_LAUNCH();
}

extern "C" int sb_embed_fwd(const void* table, const int64_t* tokens, void* out, int n, int d, int vocab,
                            void* stream) {
  if (n <= 0 || (d & 7) || !al16(table) || !al16(out)) return SB_ERR_ARG;
  embed_fwd_kernel<<<n, 128, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(table), tokens,
                                          static_cast<__nv_bfloat16*>(out), n, d, vocab);
  CHECK_LAUNCH();
}
// From tokens sorted by the caller and the positions that they had.
extern "C" int sb_embed_bwd(const void* dy, const int64_t* sorted_tok, const int64_t* perm, void* dtable, int n,
                            int d, int vocab, int accumulate, void* stream) {
  if (n <= 0 || d <= 0 || vocab <= 0 || (d & 7) || !al16(dy) || !al16(dtable)) return SB_ERR_ARG;
  const int slabs = (d / 8 + EB_THREADS - 1) / EB_THREADS;
  if (slabs > 65535) return SB_ERR_TOO_LARGE;
  const __nv_bfloat16* from = static_cast<const __nv_bfloat16*>(dy);
  __nv_bfloat16* to = static_cast<__nv_bfloat16*>(dtable);
  embed_bwd_short_runs_kernel<<<n, EB_THREADS, 0, STREAM>>>(from, sorted_tok, perm, to, n, d, vocab, accumulate);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  if (n > EB_SHORT)
    embed_bwd_long_runs_kernel<<<dim3((n - 1) / EB_SHORT + 1, slabs), EB_THREADS, 0, STREAM>>>(from, sorted_tok, perm, to, n, d, vocab, accumulate);
  CHECK_LAUNCH();
}

// From unsorted tokens. scratch: vocab + n ints.
extern "C" int sb_embed_bwd_tokens(const void* dy, const int64_t* tokens, int* scratch, void* dtable, int n, int d, int vocab,
                                   int accumulate, void* stream) {
  if (n <= 0 || vocab <= 0 || d <= 0 || (d & 7) || !al16(dy) || !al16(dtable) || !tokens || !scratch) return SB_ERR_ARG;
  const int words = d > 2048 ? 4 : d > 1024 ? 2 : 1;     // of a thread
  const int slabs = (d / 8 + EB_THREADS * words - 1) / (EB_THREADS * words);
  if (slabs > 65535) return SB_ERR_TOO_LARGE;
  int *head = scratch, *next = scratch + vocab;
  if (cudaMemsetAsync(head, 0xff, static_cast<size_t>(vocab) * sizeof(int), STREAM) != cudaSuccess) return SB_ERR_RUNTIME;
  embed_chain_kernel<<<(n + 255) / 256, 256, 0, STREAM>>>(tokens, head, next, n, vocab);
  auto kern = words == 4 ? embed_bwd_chain_kernel<4> : words == 2 ? embed_bwd_chain_kernel<2> : embed_bwd_chain_kernel<1>;
  kern<<<dim3(n, slabs), EB_THREADS, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dy), tokens, head, next,
                                                  static_cast<__nv_bfloat16*>(dtable), n, d, vocab, accumulate);
  CHECK_LAUNCH();
}
extern "C" int sb_ce_fwd_bwd(const void* logits, const int64_t* targets, float* loss_rows, void* dlogits, int rows,
                             int cols, int ld, float grad_scale, void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 7) || (ld & 7) || !al16(logits) || (dlogits && !al16(dlogits)))
    return SB_ERR_ARG;
  if (cols <= CE_THREADS * 8 * CE_KEEP) {
    ce_fwd_bwd_row_kernel<<<rows, CE_THREADS, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(logits), targets,
                                                           loss_rows, static_cast<__nv_bfloat16*>(dlogits), cols, ld,
                                                           grad_scale);
    CHECK_LAUNCH();
  }
  ce_fwd_bwd_kernel<512><<<rows, 512, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(logits), targets, loss_rows,
                                                   static_cast<__nv_bfloat16*>(dlogits), rows, cols, ld,
                                                   grad_scale);
  CHECK_LAUNCH();
}

// stats: fp32 [rows, 3] = (max, sum exp(x - max), target logit or 0) of the shard starting at vocabulary id v0.
extern "C" int sb_ce_shard_stats(const void* logits, const int64_t* targets, float* stats, int rows, int cols, int ld,
                                 int v0, void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 7) || (ld & 7) || !al16(logits)) return SB_ERR_ARG;
  ce_shard_stats_kernel<512><<<rows, 512, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(logits), targets, stats, rows,
                                                       cols, ld, v0);
  CHECK_LAUNCH();
}
// dlogits (may alias logits) = (exp(x - lse[row]) - onehot) * grad_scale for the shard's columns.
extern "C" int sb_ce_shard_grad(const void* logits, const int64_t* targets, const float* lse, void* dlogits, int rows,
                                int cols, int ld, int v0, float grad_scale, void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 7) || (ld & 7) || !al16(logits) || !al16(dlogits)) return SB_ERR_ARG;
  ce_shard_grad_kernel<<<rows, 512, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(logits), targets, lse,
                                                 static_cast<__nv_bfloat16*>(dlogits), rows, cols, ld, v0, grad_scale);
  CHECK_LAUNCH();
}

// partials: fp32 workspace of ceil(n/4096) floats.
// Partials and their sum; shared by both entry points, so that they give the same bits.
static int launch_sumsq(const void* g, size_t n, size_t nb, int is_bf16, float* partials, float* out, int accumulate,
                        cudaStream_t s) {
  const unsigned np = static_cast<unsigned>(nb), vb = static_cast<unsigned>((nb + 7) / 8);
  const __nv_bfloat16* gb = static_cast<const __nv_bfloat16*>(g);
  const float* gf = static_cast<const float*>(g);
  if (al16(g)) {
    if (is_bf16) sumsq_partial_vec_kernel<__nv_bfloat16><<<vb, 256, 0, s>>>(gb, n, np, partials);
    else sumsq_partial_vec_kernel<float><<<vb, 256, 0, s>>>(gf, n, np, partials);
  } else {
    if (is_bf16) sumsq_partial_kernel<__nv_bfloat16><<<np, 256, 0, s>>>(gb, n, partials);
    else sumsq_partial_kernel<float><<<np, 256, 0, s>>>(gf, n, partials);
  }
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  return launch_dep(sumsq_finish_kernel, dim3(1), dim3(1024), 0, s, partials, static_cast<int>(nb), out, accumulate) == cudaSuccess
             ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_sumsq(const void* g, size_t n, int is_bf16, float* partials, float* out, int accumulate,
                        void* stream) {
  if (n == 0) return SB_ERR_ARG;
  const size_t nb = (n + kSumsqElemsPerPartial - 1) / kSumsqElemsPerPartial;
  if (nb > 0x7fffffff) return SB_ERR_TOO_LARGE;
  return launch_sumsq(g, n, nb, is_bf16, partials, out, accumulate, STREAM);
}

extern "C" int sb_optim_step(float* p, float* m, float* v, const void* grad, int grad_is_bf16, void* p_bf16,
                             size_t n, size_t decay_end, float lr, float b1, float b2, float eps, float wd,
                             float bc1, float bc2, const float* grad_sumsq, float max_grad_norm, float grad_scale,
                             int mode, void* stream) {
  if (n == 0) return SB_ERR_ARG;
  const bool aligned = al16(p) && al16(m) && (mode == 2 || al16(v)) && al16(grad) &&
                       (!p_bf16 || (reinterpret_cast<uintptr_t>(p_bf16) & 7) == 0);
  const size_t n4 = aligned ? n / 4 : 0;
  const size_t first = n4 * 4;
  if (n4) {
    const unsigned blocks = static_cast<unsigned>((n4 + 255) / 256);
    const cudaError_t err =
        grad_is_bf16 ? launch_dep(optim_step_vec4_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, STREAM, p, m, v,
                                  static_cast<const __nv_bfloat16*>(grad), static_cast<__nv_bfloat16*>(p_bf16), n4, decay_end, lr,
                                  b1, b2, eps, wd, bc1, bc2, grad_sumsq, max_grad_norm, grad_scale, mode)
                     : launch_dep(optim_step_vec4_kernel<float>, dim3(blocks), dim3(256), 0, STREAM, p, m, v,
                                  static_cast<const float*>(grad), static_cast<__nv_bfloat16*>(p_bf16), n4, decay_end, lr,
                                  b1, b2, eps, wd, bc1, bc2, grad_sumsq, max_grad_norm, grad_scale, mode);
    if (err != cudaSuccess) return SB_ERR_LAUNCH;
  }
  if (first < n) {
    const unsigned blocks = static_cast<unsigned>((n - first + 255) / 256);
    if (grad_is_bf16)
      optim_step_kernel<__nv_bfloat16><<<blocks, 256, 0, STREAM>>>(
          p, m, v, static_cast<const __nv_bfloat16*>(grad), static_cast<__nv_bfloat16*>(p_bf16), first, n, decay_end,
          lr, b1, b2, eps, wd, bc1, bc2, grad_sumsq, max_grad_norm, grad_scale, mode);
    else
      optim_step_kernel<float><<<blocks, 256, 0, STREAM>>>(p, m, v, static_cast<const float*>(grad),
                                                           static_cast<__nv_bfloat16*>(p_bf16), first, n, decay_end, lr,
                                                           b1, b2, eps, wd, bc1, bc2, grad_sumsq, max_grad_norm,
                                                           grad_scale, mode);
  }
  CHECK_LAUNCH();
}

extern "C" int sb_cast(const void* in, void* out, size_t n, int to_bf16, float scale, void* stream) {
  if (n == 0) return SB_ERR_ARG;
  const unsigned blocks = static_cast<unsigned>((n + 255) / 256);
  if (to_bf16)
    cast_f32_to_bf16_kernel<<<blocks, 256, 0, STREAM>>>(static_cast<const float*>(in),
                                                        static_cast<__nv_bfloat16*>(out), n, scale);
  else
    cast_bf16_to_f32_kernel<<<blocks, 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(in),
                                                        static_cast<float*>(out), n, scale);
  CHECK_LAUNCH();
}

// Multi-tensor cast: up to MULTI_CAST_MAX fp32 tensors are rounded to bf16 into slices of one flat
// buffer in a single launch (a data-parallel bucket's gradients). blockIdx.y selects the tensor.
constexpr int MULTI_CAST_MAX = 96;
struct MultiCastParams {
  const float* src[MULTI_CAST_MAX];
  unsigned long long dst_off[MULTI_CAST_MAX];   // element offset into dst
  unsigned long long n[MULTI_CAST_MAX];
};
__global__ void multi_cast_f32_bf16_kernel(const __grid_constant__ MultiCastParams p, __nv_bfloat16* __restrict__ dst,
                                           int accumulate) {
  const int t = blockIdx.y;
  const float* __restrict__ s = p.src[t];
  __nv_bfloat16* __restrict__ d = dst + p.dst_off[t];
  const size_t n = p.n[t];
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float v = s[i];
    if (accumulate) v += __bfloat162float(d[i]);
    d[i] = __float2bfloat16_rn(v);
  }
}

// srcs / dst_offs / ns: host arrays of `count` entries (count <= 96). dst: bf16 flat buffer.
extern "C" int sb_multi_cast_f32_bf16(const void* const* srcs, const unsigned long long* dst_offs,
                                      const unsigned long long* ns, int count, void* dst, int accumulate,
                                      void* stream) {
  if (count < 1 || count > MULTI_CAST_MAX || dst == nullptr) return SB_ERR_ARG;
  MultiCastParams p;
  unsigned long long nmax = 0;
  for (int i = 0; i < count; ++i) {
    if (srcs[i] == nullptr) return SB_ERR_ARG;
    p.src[i] = static_cast<const float*>(srcs[i]);
    p.dst_off[i] = dst_offs[i];
    p.n[i] = ns[i];
    if (ns[i] > nmax) nmax = ns[i];
  }
  if (nmax == 0) return SB_ERR_ARG;
  unsigned bx = static_cast<unsigned>((nmax + 255) / 256);
  if (bx > 1024) bx = 1024;
  multi_cast_f32_bf16_kernel<<<dim3(bx, count), 256, 0, STREAM>>>(p, static_cast<__nv_bfloat16*>(dst), accumulate);
  CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// sb_sumsq_no_alloc: the sum of squares for callers that cannot allocate (see
// sumsq_no_alloc.h). Same kernels and launch shape as sb_sumsq; the per-block partials go to
// an array that is part of the library image instead of a caller-provided buffer.
// ---------------------------------------------------------------------------
#include "sumsq_no_alloc.h"
static_assert(SB_SUMSQ_NO_ALLOC_ELEMS_PER_PARTIAL == kSumsqElemsPerPartial,
              "the header's limit must describe the partial size the kernels use");

static __device__ __align__(256) float g_sumsq_no_alloc_scratch[SB_SUMSQ_NO_ALLOC_MAX_PARTIALS];

// Device address of the scratch array, resolved once per device. In host code the array's name
// is only a handle for the runtime, not something a kernel can dereference.
static float* g_sumsq_no_alloc_ptr[64] = {nullptr};

extern "C" int sb_sumsq_no_alloc(const void* g, size_t n, int is_bf16, float* out, int accumulate, void* stream) {
  if (n == 0 || g == nullptr || out == nullptr) return SB_ERR_ARG;
  if (n > SB_SUMSQ_NO_ALLOC_MAX_ELEMS) return SB_ERR_TOO_LARGE;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SB_ERR_RUNTIME;
  float* scratch = g_sumsq_no_alloc_ptr[dev];
  if (scratch == nullptr) {
    // first call on this device (which is current): ask the runtime where the array lives here
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_sumsq_no_alloc_scratch) != cudaSuccess || p == nullptr) return SB_ERR_RUNTIME;
    scratch = static_cast<float*>(p);
    g_sumsq_no_alloc_ptr[dev] = scratch;
  }
  const size_t nb = (n + kSumsqElemsPerPartial - 1) / kSumsqElemsPerPartial;
  return launch_sumsq(g, n, nb, is_bf16, scratch, out, accumulate, STREAM);
}
