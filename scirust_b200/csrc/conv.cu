// Convolutional-network kernels on NHWC bf16 activations: im2col / col2im around the tcgen05 GEMM
// (explicit-GEMM convolution forward, input gradient and weight gradient), max pooling
// forward/backward, BatchNorm2d forward/backward with running statistics, ReLU and bias helpers.
//
// Reference semantics: im2col + GEMM convolution and its adjoints
// (scirust-core/src/nn/conv2d.rs:13-208, nn/conv_utils.rs:19-120; shader IM2COL / COL2IM
// scirust-gpu/src/conv_gpu.rs:7-120 with CPU oracles :122,172), max_pool2d
// (scirust-core/src/autodiff/reverse.rs:5038), BatchNorm2d with momentum 0.1, eps 1e-5 and an
// unbiased running variance (nn/batch_norm_2d.rs:18-90,177-190).
// Layout differs from the reference on purpose: activations are [B*H*W, C] (channels innermost) so
// that a convolution's output is directly the GEMM's row-major result and per-channel statistics
// are column reductions. Patch columns are ordered (kh, kw, c) and padded to a multiple of 8.
// All reductions (col2im, column statistics) use a fixed order; no atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "api.h"

namespace sb {

int num_sms();   // gemm_tcgen05.cu

// col[(b,oh,ow), (kh,kw,c)] = x[b, oh*s - pad + kh, ow*s - pad + kw, c] (0 outside); Kp = padded width
__global__ void im2col_nhwc_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col, int B,
                                   int H, int W, int C, int KH, int KW, int stride, int pad, int OH, int OW,
                                   int Kp) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(B) * OH * OW * Kp;
  if (idx >= total) return;
  const int k = static_cast<int>(idx % Kp);
  const size_t row = idx / Kp;
  const int ow = static_cast<int>(row % OW);
  const int oh = static_cast<int>((row / OW) % OH);
  const int b = static_cast<int>(row / (static_cast<size_t>(OW) * OH));
  __nv_bfloat16 v = __float2bfloat16(0.f);
  if (k < KH * KW * C) {
    const int c = k % C;
    const int kw = (k / C) % KW;
    const int kh = k / (C * KW);
    const int ih = oh * stride - pad + kh, iw = ow * stride - pad + kw;
    if (ih >= 0 && ih < H && iw >= 0 && iw < W) v = x[((static_cast<size_t>(b) * H + ih) * W + iw) * C + c];
  }
  col[idx] = v;
}

// Division of a 31-bit value by a launch constant: one multiply-high and a shift, after Granlund and Montgomery, "Division by
// invariant integers using multiplication" (PLDI 1994): the multiplier 2^(31 + l) / d, l = ceil(log2 d), rounded up, is exact for
// n < 2^31. The index arithmetic below would otherwise spend several hundred instructions per 16-byte word on
// 64-bit divisions.
struct FastDiv {
  uint32_t d, mul, sh;
  __host__ explicit FastDiv(int div) : d(static_cast<uint32_t>(div)), mul(0), sh(0) {
    if (d <= 1) return;
    while ((1u << sh) < d) ++sh;                       // ceil(log2 d)
    mul = static_cast<uint32_t>(((1ull << (31 + sh)) + d - 1) / d);
    --sh;
  }
  __device__ __forceinline__ uint32_t div(uint32_t n) const { return d <= 1 ? n : __umulhi(n, mul) >> sh; }
  __device__ __forceinline__ uint32_t divmod(uint32_t n, uint32_t& r) const {
    const uint32_t q = div(n);
    r = n - q * d;
    return q;
  }
};

// The same gather, eight channels (16 bytes) per thread, for C a multiple of 8 (every layer but an RGB stem): bound by
// the bytes of the patch matrix it writes (86 us with 64-bit divisions for 128 x 32 x 32 x 64, 3 x 3).
__global__ void __launch_bounds__(256)
im2col_nhwc_vec8_kernel(const uint4* __restrict__ x, uint4* __restrict__ col, uint32_t total, int H, int W, int C8,
                        int taps8, int stride, int pad, FastDiv by_kp8, FastDiv by_ow, FastDiv by_oh, FastDiv by_c8,
                        FastDiv by_kw) {
  const uint32_t idx = blockIdx.x * 256u + threadIdx.x;
  if (idx >= total) return;
  uint32_t k8, ow, oh, c8, kw;
  const uint32_t row = by_kp8.divmod(idx, k8);
  const uint32_t b = by_oh.divmod(by_ow.divmod(row, ow), oh);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (k8 < static_cast<uint32_t>(taps8)) {
    const uint32_t kh = by_kw.divmod(by_c8.divmod(k8, c8), kw);
    const int ih = static_cast<int>(oh) * stride - pad + static_cast<int>(kh);
    const int iw = static_cast<int>(ow) * stride - pad + static_cast<int>(kw);
    if (ih >= 0 && ih < H && iw >= 0 && iw < W) v = __ldg(x + (static_cast<size_t>(b * H + ih) * W + iw) * C8 + c8);
  }
  col[idx] = v;
}

__device__ __forceinline__ float conv_bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float conv_bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t conv_pack(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// col2im, eight channels per thread; the taps are added in the same ascending (kh, kw) order as the scalar kernel.
// STRIDE 1 and 2 are compiled in (0: any), so that the tap test needs no division.
template <int STRIDE>
__global__ void __launch_bounds__(256)
col2im_nhwc_vec8_kernel(const uint4* __restrict__ dcol, uint4* __restrict__ dx, uint32_t total, int C8, int KH, int KW,
                        int stride_, int pad, int OH, int OW, int Kp8, FastDiv by_c8, FastDiv by_w, FastDiv by_h) {
  const uint32_t idx = blockIdx.x * 256u + threadIdx.x;
  if (idx >= total) return;
  const int stride = STRIDE ? STRIDE : stride_;
  uint32_t c8, iw, ih;
  const uint32_t b = by_h.divmod(by_w.divmod(by_c8.divmod(idx, c8), iw), ih);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int kh = 0; kh < KH; ++kh) {
    const int th = static_cast<int>(ih) + pad - kh;
    if (th < 0 || th % stride) continue;
    const int oh = th / stride;
    if (oh >= OH) continue;
    for (int kw = 0; kw < KW; ++kw) {
      const int tw = static_cast<int>(iw) + pad - kw;
      if (tw < 0 || tw % stride) continue;
      const int ow = tw / stride;
      if (ow >= OW) continue;
      const uint4 v = __ldg(dcol + (static_cast<size_t>(b * OH + oh) * OW + ow) * Kp8 + (kh * KW + kw) * C8 + c8);
      acc[0] += conv_bf_lo(v.x); acc[1] += conv_bf_hi(v.x); acc[2] += conv_bf_lo(v.y); acc[3] += conv_bf_hi(v.y);
      acc[4] += conv_bf_lo(v.z); acc[5] += conv_bf_hi(v.z); acc[6] += conv_bf_lo(v.w); acc[7] += conv_bf_hi(v.w);
    }
  }
  dx[idx] = make_uint4(conv_pack(acc[0], acc[1]), conv_pack(acc[2], acc[3]), conv_pack(acc[4], acc[5]),
                       conv_pack(acc[6], acc[7]));
}

// dx[b,ih,iw,c] = sum over (kh,kw) in ascending order of dcol[(b,oh,ow),(kh,kw,c)] where the output
// position maps onto this input pixel. Gather form: one thread per input element.
__global__ void col2im_nhwc_kernel(const __nv_bfloat16* __restrict__ dcol, __nv_bfloat16* __restrict__ dx, int B,
                                   int H, int W, int C, int KH, int KW, int stride, int pad, int OH, int OW,
                                   int Kp) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(B) * H * W * C;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % C);
  const int iw = static_cast<int>((idx / C) % W);
  const int ih = static_cast<int>((idx / (static_cast<size_t>(C) * W)) % H);
  const int b = static_cast<int>(idx / (static_cast<size_t>(C) * W * H));
  float acc = 0.f;
  for (int kh = 0; kh < KH; ++kh) {
    const int th = ih + pad - kh;
    if (th < 0 || th % stride) continue;
    const int oh = th / stride;
    if (oh >= OH) continue;
    for (int kw = 0; kw < KW; ++kw) {
      const int tw = iw + pad - kw;
      if (tw < 0 || tw % stride) continue;
      const int ow = tw / stride;
      if (ow >= OW) continue;
      acc += __bfloat162float(dcol[((static_cast<size_t>(b) * OH + oh) * OW + ow) * Kp + (kh * KW + kw) * C + c]);
    }
  }
  dx[idx] = __float2bfloat16_rn(acc);
}

// y = max over the k x k window; idx = flat offset (kh*k+kw) of the first maximum (for backward)
__global__ void maxpool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                   uint8_t* __restrict__ arg, int B, int H, int W, int C, int k, int stride, int OH,
                                   int OW) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(B) * OH * OW * C;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % C);
  const int ow = static_cast<int>((idx / C) % OW);
  const int oh = static_cast<int>((idx / (static_cast<size_t>(C) * OW)) % OH);
  const int b = static_cast<int>(idx / (static_cast<size_t>(C) * OW * OH));
  float best = -INFINITY;
  int bi = 0;
  for (int kh = 0; kh < k; ++kh)
    for (int kw = 0; kw < k; ++kw) {
      const int ih = oh * stride + kh, iw = ow * stride + kw;
      if (ih < H && iw < W) {
        const float v = __bfloat162float(x[((static_cast<size_t>(b) * H + ih) * W + iw) * C + c]);
        if (v > best) { best = v; bi = kh * k + kw; }
      }
    }
  y[idx] = __float2bfloat16_rn(best);
  if (arg) arg[idx] = static_cast<uint8_t>(bi);
}
// windows may overlap (stride < k): gather form over input pixels, fixed (kh, kw) order
__global__ void maxpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const uint8_t* __restrict__ arg,
                                   __nv_bfloat16* __restrict__ dx, int B, int H, int W, int C, int k, int stride,
                                   int OH, int OW) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(B) * H * W * C;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % C);
  const int iw = static_cast<int>((idx / C) % W);
  const int ih = static_cast<int>((idx / (static_cast<size_t>(C) * W)) % H);
  const int b = static_cast<int>(idx / (static_cast<size_t>(C) * W * H));
  float acc = 0.f;
  for (int kh = 0; kh < k; ++kh) {
    const int th = ih - kh;
    if (th < 0 || th % stride) continue;
    const int oh = th / stride;
    if (oh >= OH) continue;
    for (int kw = 0; kw < k; ++kw) {
      const int tw = iw - kw;
      if (tw < 0 || tw % stride) continue;
      const int ow = tw / stride;
      if (ow >= OW) continue;
      const size_t o = ((static_cast<size_t>(b) * OH + oh) * OW + ow) * C + c;
      if (arg[o] == kh * k + kw) acc += __bfloat162float(dy[o]);
    }
  }
  dx[idx] = __float2bfloat16_rn(acc);
}

// Column statistics of a [rows, C] matrix in two fixed-order stages.
// stage 1: partial[chunk][0][c] = sum x, partial[chunk][1][c] = sum x*y (y = x for variance, or a
// second matrix for the backward dot products). 256 rows per chunk, rows visited in order.
// MASK: elements of a count only where mask > 0 (the ReLU that followed the forward pass). The general form, for channel
// counts that are no multiple of 8 or matrices that are not aligned; sixteen rows' loads in flight, one chain of additions
// per column as ever (5000 x 13, forward and backward with ReLU: 73 us with a load at a time behind the mask, 33 so).
template <bool MASK>
__global__ void __launch_bounds__(128)
colstats_partial_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                        const __nv_bfloat16* __restrict__ mask, float* __restrict__ partial, int rows, int C) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int r0 = blockIdx.y * 256, r1 = min(rows, r0 + 256);
  float s1 = 0.f, s2 = 0.f;
  constexpr int U = 16;
  for (int r = r0; r < r1; r += U) {
    __nv_bfloat16 va[U], vb[U], vm[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const size_t at = static_cast<size_t>(min(r + i, r1 - 1)) * C + c;
      va[i] = a[at];
      vb[i] = b[at];
      if (MASK) vm[i] = mask[at];
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (r + i < r1) {
        float x = __bfloat162float(va[i]);
        if (MASK && !(__bfloat162float(vm[i]) > 0.f)) x = 0.f;
        s1 += x;
        s2 += x * __bfloat162float(vb[i]);
      }
    }
  }
  partial[(static_cast<size_t>(blockIdx.y) * 2 + 0) * C + c] = s1;
  partial[(static_cast<size_t>(blockIdx.y) * 2 + 1) * C + c] = s2;
}
__device__ __forceinline__ void conv_unpack8(const uint4& v, float (&f)[8]) {
  f[0] = conv_bf_lo(v.x); f[1] = conv_bf_hi(v.x); f[2] = conv_bf_lo(v.y); f[3] = conv_bf_hi(v.y);
  f[4] = conv_bf_lo(v.z); f[5] = conv_bf_hi(v.z); f[6] = conv_bf_lo(v.w); f[7] = conv_bf_hi(v.w);
}
__device__ __forceinline__ uint4 conv_pack8(const float (&f)[8]) {
  return make_uint4(conv_pack(f[0], f[1]), conv_pack(f[2], f[3]), conv_pack(f[4], f[5]), conv_pack(f[6], f[7]));
}
// How the gradient of a ReLU is masked by the forward output y: where y is positive, or (after an added shortcut) where y is not
// zero or below, so that a NaN in y lets the gradient through as torch's own ReLU does.
enum : int { MASK_NONE = 0, MASK_POSITIVE = 1, MASK_NOT_BELOW = 2 };
// a word of eight bf16 values where the mask of the same word of y holds, else zero
template <int MASK>
__device__ __forceinline__ uint4 conv_relu_mask8(uint4 g, const uint4& y) {
  float f[8], m[8];
  conv_unpack8(g, f);
  conv_unpack8(y, m);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = (MASK == MASK_POSITIVE ? m[j] > 0.f : !(m[j] <= 0.f)) ? f[j] : 0.f;
  return conv_pack8(f);
}

// Stage 1 of the backward sums for C a multiple of 8: bound by the bytes of the matrices. A block takes 64 columns (8 words of 16 bytes)
// of a chunk of 256 rows, 32 row lanes of 8 rows each, four rows' loads of a thread in flight; lanes, then warps are added in
// a fixed order. The one-column-per-thread kernel above walks its 256 rows in one dependent chain of 2-byte loads: 39 us
// for 131072 x 64, 8 us here. MASK_NOT_BELOW also writes the masked gradient to g_out: it is the shortcut's gradient, and the input
// gradient then reads it instead of dy and the mask.
template <int MASK>
__global__ void __launch_bounds__(256)
colstats_vec8_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, const uint4* __restrict__ mask,
                     uint4* __restrict__ g_out, float* __restrict__ partial, int rows, int C8) {
  __shared__ float s_sum[8][8][16];                 // [warp][column word][sum x: 8 | sum xy: 8]
  const int cw = threadIdx.x & 7, rl = threadIdx.x >> 3, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c8 = blockIdx.x * 8 + cw;
  const int r0 = blockIdx.y * 256 + rl;
  float s1[8], s2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s1[j] = s2[j] = 0.f;
  if (c8 < C8) {
    constexpr int U = MASK ? 4 : 8;
#pragma unroll
    for (int i0 = 0; i0 < 8; i0 += U) {
      uint4 va[U], vb[U], vm[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int r = r0 + (i0 + i) * 32;
        va[i] = vb[i] = vm[i] = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows) {
          const size_t at = static_cast<size_t>(r) * C8 + c8;
          va[i] = __ldg(a + at);
          vb[i] = __ldg(b + at);
          if (MASK) vm[i] = __ldg(mask + at);
        }
      }
#pragma unroll
      for (int i = 0; i < U; ++i) {
        if (MASK) va[i] = conv_relu_mask8<MASK>(va[i], vm[i]);
        if (MASK == MASK_NOT_BELOW) {
          const int r = r0 + (i0 + i) * 32;
          if (r < rows) g_out[static_cast<size_t>(r) * C8 + c8] = va[i];
        }
        float x[8], y[8];
        conv_unpack8(va[i], x);
        conv_unpack8(vb[i], y);
#pragma unroll
        for (int j = 0; j < 8; ++j) { s1[j] += x[j]; s2[j] += x[j] * y[j]; }
      }
    }
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s1[j] += __shfl_xor_sync(0xffffffffu, s1[j], o);
      s2[j] += __shfl_xor_sync(0xffffffffu, s2[j], o);
    }
  }
  if (lane < 8) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { s_sum[warp][cw][j] = s1[j]; s_sum[warp][cw][8 + j] = s2[j]; }
  }
  __syncthreads();
  if (threadIdx.x < 128) {
    const int w = threadIdx.x >> 4, e = threadIdx.x & 15;      // column word, (sum, column in the word)
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) v += s_sum[i][w][e];
    const int c = (blockIdx.x * 8 + w) * 8 + (e & 7);
    if (c < C8 * 8) partial[(static_cast<size_t>(blockIdx.y) * 2 + (e >> 3)) * (C8 * 8) + c] = v;
  }
}

// Stage 1 of the FORWARD statistics for even C, in the order of the kernel at the top: a column's 256 rows of a chunk in
// one chain. Mean and variance decide on which side of zero a normalised value falls, and with it the ReLU mask, so the
// order of these sums is kept to the bit; the loads are what is rearranged (a thread owns two columns and has 32 rows in
// flight, a warp reads 128 contiguous bytes per row): 39 -> 10 us for 131072 x 64; 64 in flight are level.
__global__ void __launch_bounds__(128)
colstats_chain_kernel(const uint32_t* __restrict__ a, float* __restrict__ partial, int rows, int C2) {
  const int c2 = blockIdx.x * 32 + (threadIdx.x & 31);
  const int chunk = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int r0 = chunk * 256, r1 = min(rows, r0 + 256);
  if (c2 >= C2 || r0 >= rows) return;
  const uint32_t* p = a + static_cast<size_t>(r0) * C2 + c2;
  float s1l = 0.f, s2l = 0.f, s1h = 0.f, s2h = 0.f;
  constexpr int U = 32;
  int r = r0;
  for (; r + U <= r1; r += U, p += static_cast<size_t>(U) * C2) {
    uint32_t v[U];
#pragma unroll
    for (int i = 0; i < U; ++i) v[i] = __ldg(p + static_cast<size_t>(i) * C2);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const float x = conv_bf_lo(v[i]), y = conv_bf_hi(v[i]);
      s1l += x;
      s2l += x * x;
      s1h += y;
      s2h += y * y;
    }
  }
  for (; r < r1; ++r, p += C2) {
    const uint32_t v = __ldg(p);
    const float x = conv_bf_lo(v), y = conv_bf_hi(v);
    s1l += x;
    s2l += x * x;
    s1h += y;
    s2h += y * y;
  }
  float* o = partial + static_cast<size_t>(chunk) * 4 * C2 + 2 * c2;    // [chunk][sum x | sum xx][C]
  o[0] = s1l;
  o[1] = s1h;
  o[2 * C2] = s2l;
  o[2 * C2 + 1] = s2h;
}

// Stage 2, chunks in ascending order, and what is made of a column's two sums: nothing (FIN_SUMS), mean, 1 / standard deviation and
// the running statistics of a forward pass (FIN_FORWARD: biased variance to normalise, unbiased for the running one), or the gradients
// of shift and scale (FIN_BACKWARD: dbeta = sum g, dgamma = sum g*xhat = (sum g*x - mean * sum g) * inv_std).
// Eight columns per block, so that 512 chunks are on their way at once and then added, one chain a sum, at shared-memory speed: the
// chain is what is left (131072 x 64: 5.3 us; 7.2 with 32 columns per block and 64 chunks at a time, and 1.7 to 2.6 for
// what followed in a launch of its own).
enum : int { FIN_SUMS = 0, FIN_FORWARD = 1, FIN_BACKWARD = 2 };
struct BnFinish {
  float *o1, *o2;               // FIN_SUMS: the sums; FIN_FORWARD: mean, inv_std; FIN_BACKWARD: dbeta, dgamma
  float *run_mean, *run_var;    // FIN_FORWARD, optional
  const float *mean, *inv_std;  // FIN_BACKWARD
  int rows;
  float eps, momentum;
};
// of a column's sums of x and x*x
__device__ __forceinline__ void bn_statistics(const BnFinish& f, int c, float sum, float sumsq) {
  const float n = static_cast<float>(f.rows);
  const float m = sum / n;
  const float var = fmaxf(sumsq / n - m * m, 0.f);
  f.o1[c] = m;
  f.o2[c] = rsqrtf(var + f.eps);
  if (f.run_mean) {
    f.run_mean[c] = (1.f - f.momentum) * f.run_mean[c] + f.momentum * m;
    const float unbiased = f.rows > 1 ? var * n / (n - 1.f) : var;
    f.run_var[c] = (1.f - f.momentum) * f.run_var[c] + f.momentum * unbiased;
  }
}
// of a column's sums of g and g*x
__device__ __forceinline__ void bn_gradients(const BnFinish& f, int c, float sum_g, float sum_gx) {
  f.o1[c] = sum_g;
  f.o2[c] = (sum_gx - f.mean[c] * sum_g) * f.inv_std[c];
}
constexpr int CF_COLS = 8, CF_CHUNKS = 512, CF_THREADS = 256;
template <int WHAT>
__global__ void __launch_bounds__(CF_THREADS)
colstats_finish_kernel(const float* __restrict__ partial, int chunks, int C, const BnFinish f) {
  __shared__ float s[CF_CHUNKS * 2 * CF_COLS];           // [chunk][sum x: 8 | sum xy: 8]
  constexpr int STEP = CF_THREADS / (2 * CF_COLS), PER = CF_CHUNKS / STEP;
  const int e = threadIdx.x % (2 * CF_COLS), row0 = threadIdx.x / (2 * CF_COLS);   // this thread's element of a chunk; its chunks row0 + STEP i
  const int c = blockIdx.x * CF_COLS + e % CF_COLS;
  const float* src = partial + static_cast<size_t>(e / CF_COLS) * C + c;
  float acc = 0.f;
  for (int k0 = 0; k0 < chunks; k0 += CF_CHUNKS) {
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int k = k0 + row0 + STEP * i;
      v[i] = (k < chunks && c < C) ? __ldg(src + static_cast<size_t>(k) * 2 * C) : 0.f;
    }
    __syncthreads();                                     // the chains have read the chunks before
#pragma unroll
    for (int i = 0; i < PER; ++i) s[(row0 + STEP * i) * (2 * CF_COLS) + e] = v[i];
    __syncthreads();
    if (threadIdx.x < 2 * CF_COLS) {
      const int n = min(CF_CHUNKS, chunks - k0);
#pragma unroll 16
      for (int k = 0; k < n; ++k) acc += s[k * (2 * CF_COLS) + e];
    }
  }
  if (threadIdx.x >= 32) return;                         // what is left is one warp's
  const float other = __shfl_down_sync(0xffffffffu, acc, CF_COLS);
  if (threadIdx.x >= CF_COLS || c >= C) return;
  if (WHAT == FIN_SUMS) {
    f.o1[c] = acc;
    f.o2[c] = other;
  } else if (WHAT == FIN_FORWARD) {
    bn_statistics(f, c, acc, other);
  } else {
    bn_gradients(f, c, acc, other);
  }
}

// The same from sums taken elsewhere (the C entries that begin with a layer's sums).
template <int WHAT>
__global__ void bn_from_sums_kernel(const float* __restrict__ s1, const float* __restrict__ s2, int C, const BnFinish f) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  if (WHAT == FIN_FORWARD) bn_statistics(f, c, s1[c], s2[c]);
  else bn_gradients(f, c, s1[c], s2[c]);
}
// y = (x - mean) * inv_std * gamma + beta, optional ReLU
__global__ void bn_apply_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ mean,
                                const float* __restrict__ inv_std, const float* __restrict__ gamma,
                                const float* __restrict__ beta, __nv_bfloat16* __restrict__ y, size_t total, int C,
                                int relu) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int c = static_cast<int>(i % C);
  float v = (__bfloat162float(x[i]) - mean[c]) * inv_std[c] * gamma[c] + beta[c];
  if (relu) v = fmaxf(v, 0.f);
  y[i] = __float2bfloat16_rn(v);
}
// Eight channels (16 bytes) per thread, for C a multiple of 8: bound by bytes, the per-channel values come from L1.
__device__ __forceinline__ void conv_load8(const float* __restrict__ p, float (&f)[8]) {
  const float4 u = __ldg(reinterpret_cast<const float4*>(p)), v = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w; f[4] = v.x; f[5] = v.y; f[6] = v.z; f[7] = v.w;
}
// U words of one thread lie 256 words apart: the same channels where a row's words divide 256, and the channels' values are then
// loaded once. RES adds the shortcut of a residual block before the ReLU, with the roundings and the treatment of NaN that two torch
// operators on the rounded output have. Us for 131072 x 64, one word a thread / four: 11.6 / 6.3, with a shortcut 7.9.
template <int U, bool RES>
__global__ void __launch_bounds__(256)
bn_apply_vec8_kernel(const uint4* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ inv_std,
                     const float* __restrict__ gamma, const float* __restrict__ beta, const uint4* __restrict__ res,
                     uint4* __restrict__ y, uint32_t total, FastDiv by_c8, int relu) {
  const uint32_t i0 = blockIdx.x * (256u * U) + threadIdx.x;
  if (i0 >= total) return;
  uint32_t c8;
  by_c8.divmod(i0, c8);
  uint4 xw[U], rw[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = min(i0 + u * 256u, total - 1);
    xw[u] = __ldg(x + i);
    if (RES) rw[u] = __ldg(res + i);
  }
  float m[8], s[8], g[8], b[8];
  conv_load8(mean + c8 * 8, m);
  conv_load8(inv_std + c8 * 8, s);
  conv_load8(gamma + c8 * 8, g);
  conv_load8(beta + c8 * 8, b);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u * 256u;
    if (i >= total) break;
    float v[8];
    conv_unpack8(xw[u], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = (v[j] - m[j]) * s[j] * g[j] + b[j];
      if (!RES && relu) v[j] = fmaxf(v[j], 0.f);
    }
    uint4 o = conv_pack8(v);
    if (RES) {
      float r[8];
      conv_unpack8(o, v);
      conv_unpack8(rw[u], r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = __fadd_rn(v[j], r[j]);
        if (relu && v[j] <= 0.f) v[j] = 0.f;
      }
      o = conv_pack8(v);
    }
    y[i] = o;
  }
}
// BatchNorm backward. With xhat = (x-mean)*inv_std, g = dy (already masked by ReLU when fused):
//   dbeta = sum g, dgamma = sum g*xhat, dx = gamma*inv_std/n * (n*g - dbeta - xhat*dgamma)
__global__ void bn_bwd_dx_kernel(const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ x,
                                 const float* __restrict__ mean, const float* __restrict__ inv_std,
                                 const float* __restrict__ gamma, const float* __restrict__ dgamma,
                                 const float* __restrict__ dbeta, const __nv_bfloat16* __restrict__ mask,
                                 __nv_bfloat16* __restrict__ dx, size_t total, int C, int rows) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int c = static_cast<int>(i % C);
  const float n = static_cast<float>(rows);
  const float xhat = (__bfloat162float(x[i]) - mean[c]) * inv_std[c];
  float gi = __bfloat162float(g[i]);
  if (mask && !(__bfloat162float(mask[i]) > 0.f)) gi = 0.f;
  const float v = gamma[c] * inv_std[c] / n * (n * gi - dbeta[c] - xhat * dgamma[c]);
  dx[i] = __float2bfloat16_rn(v);
}
// U as in bn_apply_vec8_kernel; the quotient of a channel is taken once a thread. Us for 131072 x 64, one word a thread / four: 15.4 / 8.4, with
// a mask 16.0 / 10.4.
template <int U, int MASK>
__global__ void __launch_bounds__(256)
bn_bwd_dx_vec8_kernel(const uint4* __restrict__ g, const uint4* __restrict__ x, const float* __restrict__ mean,
                      const float* __restrict__ inv_std, const float* __restrict__ gamma,
                      const float* __restrict__ dgamma, const float* __restrict__ dbeta,
                      const uint4* __restrict__ mask, uint4* __restrict__ dx, uint32_t total, FastDiv by_c8, int rows) {
  const uint32_t i0 = blockIdx.x * (256u * U) + threadIdx.x;
  if (i0 >= total) return;
  uint32_t c8;
  by_c8.divmod(i0, c8);
  const float n = static_cast<float>(rows);
  uint4 gw[U], xw[U], mw[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = min(i0 + u * 256u, total - 1);
    gw[u] = __ldg(g + i);
    xw[u] = __ldg(x + i);
    if (MASK) mw[u] = __ldg(mask + i);
  }
  float m[8], s[8], k[8], dg[8], db[8];
  conv_load8(mean + c8 * 8, m);
  conv_load8(inv_std + c8 * 8, s);
  conv_load8(gamma + c8 * 8, k);
  conv_load8(dgamma + c8 * 8, dg);
  conv_load8(dbeta + c8 * 8, db);
#pragma unroll
  for (int j = 0; j < 8; ++j) k[j] = k[j] * s[j] / n;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u * 256u;
    if (i >= total) break;
    if (MASK) gw[u] = conv_relu_mask8<MASK>(gw[u], mw[u]);
    float gi[8], xi[8];
    conv_unpack8(gw[u], gi);
    conv_unpack8(xw[u], xi);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float xhat = (xi[j] - m[j]) * s[j];
      gi[j] = k[j] * (n * gi[j] - db[j] - xhat * dg[j]);
    }
    dx[i] = conv_pack8(gi);
  }
}
// g = dy * (y > 0)
__global__ void relu_mask_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ y,
                                 __nv_bfloat16* __restrict__ g, size_t total) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  g[i] = __bfloat162float(y[i]) > 0.f ? dy[i] : __float2bfloat16(0.f);
}
// y = act(x + bias[c])
__global__ void bias_act_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ bias,
                                __nv_bfloat16* __restrict__ y, size_t total, int C, int relu) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  float v = __bfloat162float(x[i]) + (bias ? bias[i % C] : 0.f);
  if (relu) v = fmaxf(v, 0.f);
  y[i] = __float2bfloat16_rn(v);
}

}  // namespace sb

using namespace sb;
#define STREAM static_cast<cudaStream_t>(stream)
#define CHECK_LAUNCH() return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH
static inline bool conv_al16(const void* a, const void* b, const void* c = nullptr, const void* d = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}
static inline unsigned nblk(size_t n) { return static_cast<unsigned>((n + 255) / 256); }

extern "C" int sb_im2col_nhwc(const void* x, void* col, int B, int H, int W, int C, int KH, int KW, int stride,
                              int pad, int OH, int OW, int Kp, void* stream) {
  if (B <= 0 || Kp < KH * KW * C || (Kp & 7)) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(B) * OH * OW * Kp;
  if ((C & 7) == 0 && total / 8 <= 0x7fffff00u && conv_al16(x, col)) {
    im2col_nhwc_vec8_kernel<<<nblk(total / 8), 256, 0, STREAM>>>(
        static_cast<const uint4*>(x), static_cast<uint4*>(col), static_cast<uint32_t>(total / 8), H, W, C / 8,
        KH * KW * (C / 8), stride, pad, FastDiv(Kp / 8), FastDiv(OW), FastDiv(OH), FastDiv(C / 8), FastDiv(KW));
    CHECK_LAUNCH();
  }
  im2col_nhwc_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(x),
                                                      static_cast<__nv_bfloat16*>(col), B, H, W, C, KH, KW, stride,
                                                      pad, OH, OW, Kp);
  CHECK_LAUNCH();
}
extern "C" int sb_col2im_nhwc(const void* dcol, void* dx, int B, int H, int W, int C, int KH, int KW, int stride,
                              int pad, int OH, int OW, int Kp, void* stream) {
  if (B <= 0 || Kp < KH * KW * C) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(B) * H * W * C;
  if ((C & 7) == 0 && (Kp & 7) == 0 && total / 8 <= 0x7fffff00u && conv_al16(dcol, dx)) {
    auto kern = stride == 1 ? col2im_nhwc_vec8_kernel<1> : stride == 2 ? col2im_nhwc_vec8_kernel<2> : col2im_nhwc_vec8_kernel<0>;
    kern<<<nblk(total / 8), 256, 0, STREAM>>>(static_cast<const uint4*>(dcol), static_cast<uint4*>(dx),
                                              static_cast<uint32_t>(total / 8), C / 8, KH, KW, stride, pad, OH, OW,
                                              Kp / 8, FastDiv(C / 8), FastDiv(W), FastDiv(H));
    CHECK_LAUNCH();
  }
  col2im_nhwc_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dcol),
                                                      static_cast<__nv_bfloat16*>(dx), B, H, W, C, KH, KW, stride,
                                                      pad, OH, OW, Kp);
  CHECK_LAUNCH();
}
extern "C" int sb_maxpool_fwd(const void* x, void* y, void* arg, int B, int H, int W, int C, int k, int stride,
                              int OH, int OW, void* stream) {
  if (B <= 0 || k <= 0 || k > 15) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(B) * OH * OW * C;
  maxpool_fwd_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(x),
                                                      static_cast<__nv_bfloat16*>(y), static_cast<uint8_t*>(arg), B,
                                                      H, W, C, k, stride, OH, OW);
  CHECK_LAUNCH();
}
extern "C" int sb_maxpool_bwd(const void* dy, const void* arg, void* dx, int B, int H, int W, int C, int k,
                              int stride, int OH, int OW, void* stream) {
  if (B <= 0 || k <= 0) return SB_ERR_ARG;
  const size_t total = static_cast<size_t>(B) * H * W * C;
  maxpool_bwd_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dy),
                                                      static_cast<const uint8_t*>(arg),
                                                      static_cast<__nv_bfloat16*>(dx), B, H, W, C, k, stride, OH, OW);
  CHECK_LAUNCH();
}
// Whether the kernels of eight channels a thread take a [rows, C] matrix (addresses aside).
static bool bn_vec8(size_t total, int C) { return (C & 7) == 0 && total / 8 <= 0x7fffff00u; }
// Words of a thread: see bn_apply_vec8_kernel. A small matrix keeps one, so that its words reach all SMs (four blocks of 256 on each).
static int bn_words(size_t total, int C) {
  return 256 % (C / 8) == 0 && total / 8 >= 4u * num_sms() * 4 * 256 ? 4 : 1;
}

// Column sums of a and of a * b into `partial` (2 * ceil(rows/256) * C floats) and what WHAT makes of them. g_out: see colstats_vec8_kernel.
template <int WHAT>
static int colstats(const void* a, const void* b, const void* mask, void* g_out, float* partial, const BnFinish& f, int rows, int C,
                    cudaStream_t stream) {
  const int chunks = (rows + 255) / 256;
  const uint4 *a4 = static_cast<const uint4*>(a), *b4 = static_cast<const uint4*>(b), *m4 = static_cast<const uint4*>(mask);
  const bool vec8 = (C & 7) == 0 && chunks <= 65535 && conv_al16(a, b, mask, g_out);
  if (g_out && !vec8) return SB_ERR_ARG;
  if (a == b && !mask && (C & 1) == 0 && (reinterpret_cast<uintptr_t>(a) & 3) == 0 && (chunks + 3) / 4 <= 65535) {
    colstats_chain_kernel<<<dim3((C / 2 + 31) / 32, (chunks + 3) / 4), 128, 0, stream>>>(static_cast<const uint32_t*>(a),
                                                                                        partial, rows, C / 2);
  } else if (vec8) {
    const dim3 grid((C / 8 + 7) / 8, chunks);
    auto kern = g_out ? colstats_vec8_kernel<MASK_NOT_BELOW> : mask ? colstats_vec8_kernel<MASK_POSITIVE> : colstats_vec8_kernel<MASK_NONE>;
    kern<<<grid, 256, 0, stream>>>(a4, b4, m4, static_cast<uint4*>(g_out), partial, rows, C / 8);
  } else {
    dim3 grid((C + 127) / 128, chunks);
    auto kern = mask ? colstats_partial_kernel<true> : colstats_partial_kernel<false>;
    kern<<<grid, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b),
                                   static_cast<const __nv_bfloat16*>(mask), partial, rows, C);
  }
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  colstats_finish_kernel<WHAT><<<(C + CF_COLS - 1) / CF_COLS, CF_THREADS, 0, stream>>>(partial, chunks, C, f);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}
static int bn_apply(const void* x, const float* mean, const float* inv_std, const float* gamma, const float* beta,
                    const void* res, void* y, int rows, int C, int relu, cudaStream_t stream) {
  const size_t total = static_cast<size_t>(rows) * C;
  if (bn_vec8(total, C) && conv_al16(x, y, res) && conv_al16(mean, inv_std, gamma, beta)) {
    const int u = bn_words(total, C);
    auto kern = u == 4 ? (res ? bn_apply_vec8_kernel<4, true> : bn_apply_vec8_kernel<4, false>)
                       : (res ? bn_apply_vec8_kernel<1, true> : bn_apply_vec8_kernel<1, false>);
    kern<<<nblk((total / 8 + u - 1) / u), 256, 0, stream>>>(static_cast<const uint4*>(x), mean, inv_std, gamma, beta,
                                                            static_cast<const uint4*>(res), static_cast<uint4*>(y),
                                                            static_cast<uint32_t>(total / 8), FastDiv(C / 8), relu);
    CHECK_LAUNCH();
  }
  if (res) return SB_ERR_ARG;
  bn_apply_kernel<<<nblk(total), 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), mean, inv_std, gamma, beta,
                                                   static_cast<__nv_bfloat16*>(y), total, C, relu);
  CHECK_LAUNCH();
}
static int bn_bwd_dx(const void* g, const void* x, const float* mean, const float* inv_std, const float* gamma,
                     const float* dgamma, const float* dbeta, const void* mask, void* dx, int rows, int C, cudaStream_t stream) {
  const size_t total = static_cast<size_t>(rows) * C;
  if (bn_vec8(total, C) && conv_al16(g, x, dx, mask) && conv_al16(mean, inv_std, gamma) && conv_al16(dgamma, dbeta)) {
    const int u = bn_words(total, C);
    auto kern = u == 4 ? (mask ? bn_bwd_dx_vec8_kernel<4, MASK_POSITIVE> : bn_bwd_dx_vec8_kernel<4, MASK_NONE>)
                       : (mask ? bn_bwd_dx_vec8_kernel<1, MASK_POSITIVE> : bn_bwd_dx_vec8_kernel<1, MASK_NONE>);
    kern<<<nblk((total / 8 + u - 1) / u), 256, 0, stream>>>(
        static_cast<const uint4*>(g), static_cast<const uint4*>(x), mean, inv_std, gamma, dgamma, dbeta,
        static_cast<const uint4*>(mask), static_cast<uint4*>(dx), static_cast<uint32_t>(total / 8), FastDiv(C / 8), rows);
    CHECK_LAUNCH();
  }
  bn_bwd_dx_kernel<<<nblk(total), 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(g),
                                                    static_cast<const __nv_bfloat16*>(x), mean, inv_std, gamma,
                                                    dgamma, dbeta, static_cast<const __nv_bfloat16*>(mask),
                                                    static_cast<__nv_bfloat16*>(dx), total, C, rows);
  CHECK_LAUNCH();
}
// s1 = column sums of a, s2 = of a * b; `mask` (optional, same shape): elements of a count where mask > 0.
// partial: 2 * ceil(rows/256) * C floats
extern "C" int sb_colstats_masked(const void* a, const void* b, const void* mask, float* partial, float* s1, float* s2,
                                  int rows, int C, void* stream) {
  if (rows <= 0 || C <= 0) return SB_ERR_ARG;
  BnFinish f = {};
  f.o1 = s1; f.o2 = s2;
  return colstats<FIN_SUMS>(a, b, mask, nullptr, partial, f, rows, C, STREAM);
}
extern "C" int sb_bn_fwd(const void* x, const float* sum, const float* sumsq, const float* gamma, const float* beta,
                         float* mean, float* inv_std, float* run_mean, float* run_var, void* y, int rows, int C,
                         float eps, float momentum, int relu, int training, void* stream) {
  if (rows <= 0 || C <= 0) return SB_ERR_ARG;
  if (training) {
    BnFinish f = {};
    f.o1 = mean; f.o2 = inv_std; f.run_mean = run_mean; f.run_var = run_var;
    f.rows = rows; f.eps = eps; f.momentum = momentum;
    bn_from_sums_kernel<FIN_FORWARD><<<(C + 127) / 128, 128, 0, STREAM>>>(sum, sumsq, C, f);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  }
  return bn_apply(x, mean, inv_std, gamma, beta, nullptr, y, rows, C, relu, STREAM);
}
// The forward pass of a layer: with `partial` (2 * ceil(rows/256) * C floats) on the batch's own statistics, which are written to mean
// and inv_std and into the running ones (optional); without it mean and inv_std are given. res (optional, C a multiple of 8, 16-byte
// aligned like the other tensors, else SB_ERR_ARG): a shortcut that is added before the ReLU.
extern "C" int sb_bn_layer_fwd(const void* x, float* partial, const float* gamma, const float* beta, float* mean, float* inv_std,
                               float* run_mean, float* run_var, const void* res, void* y, int rows, int C, float eps,
                               float momentum, int relu, void* stream) {
  if (rows <= 0 || C <= 0) return SB_ERR_ARG;
  if (res && !(bn_vec8(static_cast<size_t>(rows) * C, C) && conv_al16(x, y, res) && conv_al16(mean, inv_std, gamma, beta)))
    return SB_ERR_ARG;
  if (partial) {
    BnFinish f = {};
    f.o1 = mean; f.o2 = inv_std; f.run_mean = run_mean; f.run_var = run_var;
    f.rows = rows; f.eps = eps; f.momentum = momentum;
    const int rc = colstats<FIN_FORWARD>(x, x, nullptr, nullptr, partial, f, rows, C, STREAM);
    if (rc) return rc;
  }
  return bn_apply(x, mean, inv_std, gamma, beta, res, y, rows, C, relu, STREAM);
}
// Its backward pass. mask (optional): the forward output after a fused ReLU; dy counts where it is positive. g_out (optional, with a
// mask; C a multiple of 8 and all tensors 16-byte aligned, else SB_ERR_ARG): the masked dy, the gradient of an added shortcut.
extern "C" int sb_bn_layer_bwd(const void* dy, const void* x, const void* mask, void* g_out, float* partial, const float* mean,
                               const float* inv_std, const float* gamma, float* dgamma, float* dbeta, void* dx, int rows, int C,
                               void* stream) {
  if (rows <= 0 || C <= 0 || (g_out && !mask)) return SB_ERR_ARG;
  BnFinish f = {};
  f.o1 = dbeta; f.o2 = dgamma; f.mean = mean; f.inv_std = inv_std;
  const int rc = colstats<FIN_BACKWARD>(dy, x, mask, g_out, partial, f, rows, C, STREAM);
  if (rc) return rc;
  return bn_bwd_dx(g_out ? g_out : dy, x, mean, inv_std, gamma, dgamma, dbeta, g_out ? nullptr : mask, dx, rows, C, STREAM);
}
// mask (optional): the forward output after a fused ReLU; g counts where it is positive (sum_g, sum_gx likewise).
extern "C" int sb_bn_bwd_masked(const void* g, const void* x, const float* sum_g, const float* sum_gx,
                                const float* mean, const float* inv_std, const float* gamma, float* dgamma,
                                float* dbeta, const void* mask, void* dx, int rows, int C, void* stream) {
  if (rows <= 0 || C <= 0) return SB_ERR_ARG;
  BnFinish f = {};
  f.o1 = dbeta; f.o2 = dgamma; f.mean = mean; f.inv_std = inv_std;
  bn_from_sums_kernel<FIN_BACKWARD><<<(C + 127) / 128, 128, 0, STREAM>>>(sum_g, sum_gx, C, f);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  return bn_bwd_dx(g, x, mean, inv_std, gamma, dgamma, dbeta, mask, dx, rows, C, STREAM);
}
// The forms without a mask: entry points of their own in the C ABI. The layers above begin with sb_bn_layer_fwd / _bwd, hosts of the C ABI
// that take the sums themselves (synchronised over ranks, say) with these.
extern "C" int sb_colstats(const void* a, const void* b, float* partial, float* s1, float* s2, int rows, int C,
                           void* stream) {
  return sb_colstats_masked(a, b, nullptr, partial, s1, s2, rows, C, stream);
}
extern "C" int sb_bn_bwd(const void* g, const void* x, const float* sum_g, const float* sum_gx, const float* mean,
                         const float* inv_std, const float* gamma, float* dgamma, float* dbeta, void* dx, int rows,
                         int C, void* stream) {
  return sb_bn_bwd_masked(g, x, sum_g, sum_gx, mean, inv_std, gamma, dgamma, dbeta, nullptr, dx, rows, C, stream);
}
extern "C" int sb_relu_mask(const void* dy, const void* y, void* g, size_t total, void* stream) {
  if (total == 0) return SB_ERR_ARG;
  relu_mask_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(dy),
                                                    static_cast<const __nv_bfloat16*>(y),
                                                    static_cast<__nv_bfloat16*>(g), total);
  CHECK_LAUNCH();
}
extern "C" int sb_bias_act(const void* x, const float* bias, void* y, size_t total, int C, int relu, void* stream) {
  if (total == 0 || C <= 0) return SB_ERR_ARG;
  bias_act_kernel<<<nblk(total), 256, 0, STREAM>>>(static_cast<const __nv_bfloat16*>(x), bias,
                                                   static_cast<__nv_bfloat16*>(y), total, C, relu);
  CHECK_LAUNCH();
}
