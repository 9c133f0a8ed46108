// RoPE over the rows of a fused projection [q heads | k heads | v heads], in place, and with KV the copy of the rotated k heads and
// of the v heads into a paged cache. Interleaved pairs, head-local frequency; table: cos / sin fp32 [max_pos, dh/2]; sign -1 is the
// backward pass (the transpose of a rotation is the rotation by the negative angle).
//
// Bound by the bytes of the heads: in large calls a thread owns eight columns of a head (16 bytes) in RR_HEADS heads of one row, so
// the table is read once for all of them and their loads are on their way together; small ones take a thread per word. One head a
// thread, found by a 64-bit division: 16384 rows, 20 heads of 64: 20.5 us, 12.8 so; 2048 rows, 40 heads of 128 and the copy to the
// cache: 10.4 + 4.9 / 9.2.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sb {

constexpr int RR_HEADS = 4, RR_THREADS = 256;

struct RopeRows {
  __nv_bfloat16* x;
  int ld, rows, rot_heads, heads, dh;       // the first rot_heads of heads rotate
  int seq_len, offset;                      // position of row r: positions[r] if given, else r % seq_len + offset
  const int* positions;
  const float *cos_t, *sin_t;
  float sign;
  // KV: heads [q_heads, q_heads + kv_heads) are keys, the next kv_heads values
  int q_heads, kv_heads, page, max_blocks;
  __nv_bfloat16* pool;                      // [blocks, 2, kv_heads, page, dh]
  const int *block_table, *seq_of;
};

__device__ __forceinline__ uint32_t rr_rotate(uint32_t v, float c, float s) {
  const float x0 = __uint_as_float(v << 16), x1 = __uint_as_float(v & 0xffff0000u);
  // which product is rounded is spelt out, so that it does not change with the code around it
  const __nv_bfloat162 h = __floats2bfloat162_rn(__fmaf_rn(x0, c, -__fmul_rn(x1, s)), __fmaf_rn(x1, c, __fmul_rn(x0, s)));
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void rr_to_cache(const RopeRows& p, int r, int pos, int h, int qd, const uint4& v) {
  const int kv = h >= p.q_heads + p.kv_heads ? 1 : 0, hk = h - p.q_heads - kv * p.kv_heads;
  const int blk = p.block_table[p.seq_of[r] * p.max_blocks + pos / p.page];
  *(reinterpret_cast<uint4*>(p.pool + (((static_cast<size_t>(blk) * 2 + kv) * p.kv_heads + hk) * p.page + pos % p.page) * p.dh) + qd) = v;
}

template <bool KV>
__global__ void __launch_bounds__(RR_THREADS) rope_rows_kernel(const RopeRows p) {
  const int q8 = p.dh >> 3;                                     // 16-byte words of a head
  const int per_block = q8 < RR_THREADS ? RR_THREADS / q8 : 1;  // rows of a CTA
  const int local = q8 < RR_THREADS ? static_cast<int>(threadIdx.x) / q8 : 0;
  if (local >= per_block) return;
  const long long row_ = static_cast<long long>(blockIdx.x) * per_block + local;
  if (row_ >= p.rows) return;
  const int r = static_cast<int>(row_), h0 = blockIdx.y * RR_HEADS, half = p.dh >> 1;
  const int pos = p.positions ? p.positions[r] : r % p.seq_len + p.offset;
  for (int qd = static_cast<int>(threadIdx.x) - local * q8; qd < q8; qd += RR_THREADS) {
    uint4* at = reinterpret_cast<uint4*>(p.x + static_cast<size_t>(r) * p.ld) + static_cast<size_t>(h0) * q8 + qd;
    uint4 v[RR_HEADS];
#pragma unroll
    for (int u = 0; u < RR_HEADS; ++u)
      if (h0 + u < p.heads) v[u] = at[u * q8];
    const size_t row_t = static_cast<size_t>(pos) * half + qd * 4;
    const float4 c = *reinterpret_cast<const float4*>(p.cos_t + row_t);
    float4 s = *reinterpret_cast<const float4*>(p.sin_t + row_t);
    s.x *= p.sign; s.y *= p.sign; s.z *= p.sign; s.w *= p.sign;
#pragma unroll
    for (int u = 0; u < RR_HEADS; ++u) {
      const int h = h0 + u;
      if (h >= p.heads) break;
      if (h < p.rot_heads) {
        v[u].x = rr_rotate(v[u].x, c.x, s.x); v[u].y = rr_rotate(v[u].y, c.y, s.y);
        v[u].z = rr_rotate(v[u].z, c.z, s.z); v[u].w = rr_rotate(v[u].w, c.w, s.w);
        at[u * q8] = v[u];
      }
      if (KV && h >= p.q_heads) rr_to_cache(p, r, pos, h, qd, v[u]);
    }
  }
}

// The same with one word of 16 bytes a thread, in the order of memory: more threads with less to do each.
template <bool KV>
__global__ void __launch_bounds__(RR_THREADS) rope_words_kernel(const RopeRows p) {
  const int q8 = p.dh >> 3, words = p.heads * q8;
  const uint32_t total = static_cast<uint32_t>(p.rows) * words, i = blockIdx.x * RR_THREADS + threadIdx.x;
  if (i >= total) return;
  const int r = static_cast<int>(i / words), w = static_cast<int>(i) - r * words, h = w / q8, qd = w - h * q8;
  const int pos = p.positions ? p.positions[r] : r % p.seq_len + p.offset;
  uint4* at = reinterpret_cast<uint4*>(p.x + static_cast<size_t>(r) * p.ld) + w;
  uint4 v = *at;
  if (h < p.rot_heads) {
    const size_t row_t = static_cast<size_t>(pos) * (p.dh >> 1) + qd * 4;
    const float4 c = *reinterpret_cast<const float4*>(p.cos_t + row_t);
    float4 s = *reinterpret_cast<const float4*>(p.sin_t + row_t);
    s.x *= p.sign; s.y *= p.sign; s.z *= p.sign; s.w *= p.sign;
    v.x = rr_rotate(v.x, c.x, s.x); v.y = rr_rotate(v.y, c.y, s.y);
    v.z = rr_rotate(v.z, c.z, s.z); v.w = rr_rotate(v.w, c.w, s.w);
    *at = v;
  }
  if (KV && h >= p.q_heads) rr_to_cache(p, r, pos, h, qd, v);
}

int num_sms();   // gemm_tcgen05.cu

// Which of the two. Words while the GPU holds a thread for each of them at once, for one head, which has nothing to share, and for head
// dimensions below 32, where a thread's heads lie too close for whole sectors. Us, heads x words / words: 64 rows of 20 heads of 64 2.24 /
// 1.82, 999 of 5 of 128 2.24 / 2.12, 16384 of 1 of 256 5.72 / 4.59, of 20 of 8 6.33 / 3.55; but 4096 of 8 of 128 3.57 / 4.51, 16384 of
// 20 of 64 9.30 / 15.06. With the cache, 333 rows of 48 heads of 128 3.36 / 3.06, 2048 7.57 / 9.74.
template <bool KV>
static cudaError_t launch_rope_rows(const RopeRows& p, cudaStream_t stream) {
  const int q8 = p.dh >> 3, per_block = q8 < RR_THREADS ? RR_THREADS / q8 : 1;
  const long long words = static_cast<long long>(p.rows) * p.heads * q8;
  if (words <= 2048ll * num_sms() || ((p.heads == 1 || p.dh < 32) && words < 0x7fffff00ll)) {
    rope_words_kernel<KV><<<static_cast<unsigned>((words + RR_THREADS - 1) / RR_THREADS), RR_THREADS, 0, stream>>>(p);
    return cudaGetLastError();
  }
  rope_rows_kernel<KV><<<dim3(static_cast<unsigned>((static_cast<long long>(p.rows) + per_block - 1) / per_block), (p.heads + RR_HEADS - 1) / RR_HEADS),
                         RR_THREADS, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace sb
