// GQA flash-attention backward for sm_100a on tcgen05 tensor cores, without atomics.
//
// Three launches:
//   1. delta[b,h,s] = sum_d dO * O                                   (bandwidth-bound)
//   2. dK/dV: one CTA per (128-row kv tile, kv head, batch); loops over the query heads of
//      the group and over query tiles in ascending order, accumulating dK and dV in tensor
//      memory:  S^T = K Q^T,  dP^T = V dO^T,  dV += P^T dO,  dK += dS^T Q
//   3. dQ: one CTA per (128-row query tile, head, batch); loops over kv tiles in ascending
//      order:   S = Q K^T,  dP = dO V^T,  dQ += dS K
// Every sum has a fixed order, so gradients are bitwise repeatable (the reference gets the
// same property from per-(sequence, head) serial launches: cuda_model.rs:948-999, and
// softmax_bwd / scale_mask_bwd in scirust-cuda/src/chain.rs:479,337).
//
// P is recomputed from the saved log-sum-exp; dS = P * (dP - delta) * scale.
#include "sm100_ptx.cuh"
#include "api.h"
#include "per_device.h"

namespace sb {

int make_tmap_3d_bf16(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t pitch1,
                      uint64_t pitch2, uint32_t box0, uint32_t box1);
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

constexpr int BT = 128;          // tile edge (query rows and kv rows)
constexpr int BWD_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 softmax (two per TMEM lane quarter)
constexpr float LOG2E = 1.4426950408889634f;

struct BwdParams {
  int B, S, H, Hkv;
  int ld_dqkv;
  float scale, scale_log2;
  int causal;
  const float* lse;    // [B,H,S]
  const float2* stats; // [B,H,S] (lse * log2(e), delta), written by attn_delta_kernel
  __nv_bfloat16* dqkv; // [B*S, ld_dqkv]
  int* status;
  int spill_ds;        // dK/dV kernel also stores every dS tile to the [B*H, S, S] scratch (see dQ below)
};

// Store 32 bf16 (packed in 16 words) of row r, columns [c*32, c*32+32) into a [128 x 128] bf16 tile
// laid out as two 128-byte-swizzled K-major chunks of 64 columns.
__device__ __forceinline__ void store_row32_sw128(uint8_t* tile, int r, int c, const uint32_t* pk) {
  uint8_t* prow = tile + (c >> 1) * (BT * 128) + r * 128;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int unit = ((c & 1) * 4 + u) ^ (r & 7);
    *reinterpret_cast<uint4*>(prow + unit * 16) = make_uint4(pk[u * 4], pk[u * 4 + 1], pk[u * 4 + 2], pk[u * 4 + 3]);
  }
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Element-wise core of the recomputing dQ kernel for 32 score columns of one query row (thread = query
// row r, TMEM lane r): p = 2^(s*sl2 - lse2), dS = p * (dP*scale - delta*scale); columns beyond
// `lim` are masked. Writes dS as bf16 into the swizzled [q x kv] tile.
template <bool MASK>
__device__ __forceinline__ void bwd_chunk(uint32_t tm_S, uint32_t tm_dP, uint32_t lane_off, int c, int r, int lim,
                                          float sl2, float lse2, float delta_s, float scale, uint8_t* ds_buf) {
  uint32_t sv[32], dv[32];
  tmem_ld_32x32(tm_S + lane_off + c * 32, sv);
  tmem_ld_32x32(tm_dP + lane_off + c * 32, dv);
  tmem_ld_wait();
  uint32_t dk[16];
  const float neg_lse2 = -lse2, neg_delta = -delta_s;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    // packed pairs: (s0, s1) * sl2 - lse2, (dP0, dP1) * scale - delta * scale, p * (...)
    fma2(sv[i], sv[i + 1], sl2, neg_lse2);
    fma2(dv[i], dv[i + 1], scale, neg_delta);
    float p0 = fast_exp2(__uint_as_float(sv[i]));
    float p1 = fast_exp2(__uint_as_float(sv[i + 1]));
    if (MASK) {
      if (c * 32 + i > lim) p0 = 0.f;
      if (c * 32 + i + 1 > lim) p1 = 0.f;
    }
    mul2(dv[i], dv[i + 1], p0, p1);
    dk[i >> 1] = pack_bf16x2(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1]));
  }
  store_row32_sw128(ds_buf, r, c, dk);
}

// Row statistics of the backward pass, (lse * log2(e), delta = rowsum(dO * O)) for every head and row. Bound by the bytes of O and dO: a
// CTA takes eight rows x 512 columns, a row per warp; a group of dh/8 lanes (8 or 16) adds up its head in a butterfly, and
// the results leave through shared memory, so that the statistics of a head, which lie S apart from the next head's, are read and
// written eight rows at a time. With a group per (row, head), a 64-bit division each and scattered statistics 2 x 2048 x 32
// heads of 128 took 19.7 us, 14.2 so (four rows a warp: 16.9); 8 x 2048 x 16 heads of 64 22.3 / 16.9.
constexpr int DL_ROWS = 8, DL_COLS = 512;
__global__ void __launch_bounds__(DL_ROWS * 32)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse,
                  float2* __restrict__ stats, int rows, int S, int H, int dh, int ld_o, int ld_do) {
  __shared__ float s_delta[DL_COLS / 64][DL_ROWS + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = dh >> 3;
  const int row0 = blockIdx.x * DL_ROWS, col0 = blockIdx.y * DL_COLS, cols = H * dh;
  uint4 a[2], g[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = col0 + i * 256 + lane * 8;
    a[i] = g[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row0 + warp < rows && c < cols) {
      a[i] = __ldg(reinterpret_cast<const uint4*>(o + static_cast<size_t>(row0 + warp) * ld_o + c));
      g[i] = __ldg(reinterpret_cast<const uint4*>(d_o + static_cast<size_t>(row0 + warp) * ld_do + c));
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint4 x = a[i], y = g[i];
    float acc = bf16_lo(x.x) * bf16_lo(y.x) + bf16_hi(x.x) * bf16_hi(y.x) + bf16_lo(x.y) * bf16_lo(y.y) +
                bf16_hi(x.y) * bf16_hi(y.y) + bf16_lo(x.z) * bf16_lo(y.z) + bf16_hi(x.z) * bf16_hi(y.z) +
                bf16_lo(x.w) * bf16_lo(y.w) + bf16_hi(x.w) * bf16_hi(y.w);
    for (int off = gl >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane % gl == 0) s_delta[(i * 256 + lane * 8) / dh][warp] = acc;
  }
  __syncthreads();
  const int hl = threadIdx.x / DL_ROWS, rl = threadIdx.x % DL_ROWS;     // head of this slab, row of this CTA
  const int h = col0 / dh + hl, row = row0 + rl;
  if (hl < DL_COLS / dh && h < H && row < rows) {
    const int b = row / S;
    const size_t idx = (static_cast<size_t>(b) * H + h) * S + (row - b * S);
    stats[idx] = make_float2(lse[idx] * LOG2E, s_delta[hl][rl]);
  }
}

// --------------------------------------------------------------------------- dK / dV
// Pipeline at head dimension 64. A softmax thread takes its scores and dP into registers at once, so S and dP of iteration
// t+1 follow while the exponentials of t run, and the gradient products of t while those of t+1 do: an iteration is as
// long as its softmax. That takes three (Q, dO) stages, and P^T in one buffer to make room for them (dV(t-1) has read it
// long before P(t) is ready); dS^T keeps two, since its bulk store reads it too. The issuing warp walks through its loop as
// a whole with one lane issuing, so that descriptors stay in uniform registers: as a single thread it needed 1600 cycles
// for the 16 gradient products, which run in 900. Until then the scores of t+1 waited for the whole softmax of t, then for a
// stage, and then for the issuer, 3500 cycles an iteration: 8 x 2048 tokens of 16 heads, causal, the whole backward 449 us,
// 375 now (with the dQ stream below). At 128 shared memory has no room for this: the kernel below this one.
struct DkvCfg {
  static constexpr int DH = 64;
  static constexpr int NPB = 2;                       // dS^T buffers
  static constexpr int QS = 3;                        // (Q, dO) ring stages
  static constexpr int T_BYTES = BT * DH * 2;         // one [128 x DH] tile
  static constexpr int PT_BYTES = BT * BT * 2;
  static constexpr int TILE_BYTES = 2 * T_BYTES + QS * 2 * T_BYTES + (1 + NPB) * PT_BYTES;
  static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 128;
  static constexpr int TMEM_COLS = 512;  // S^T 128 | dP^T 128 | dK DH | dV DH
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
};

__global__ void __launch_bounds__(BWD_THREADS, 1)
attention_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                         const __grid_constant__ CUtensorMap tm_ds, const BwdParams p) {
  using Cfg = DkvCfg;
  constexpr int DH = Cfg::DH, NCH = DH / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::T_BYTES;
  uint8_t* sQ = sV + Cfg::T_BYTES;                 // QS stages
  uint8_t* sdO = sQ + Cfg::QS * Cfg::T_BYTES;      // QS stages
  uint8_t* sPT = sdO + Cfg::QS * Cfg::T_BYTES;
  uint8_t* sdST = sPT + Cfg::PT_BYTES;             // NPB buffers
  uint64_t* bars = reinterpret_cast<uint64_t*>(sdST + Cfg::NPB * Cfg::PT_BYTES);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;            // QS
  uint64_t* q_empty = q_full + Cfg::QS;   // QS
  uint64_t* st_full = q_empty + Cfg::QS;
  uint64_t* st_free = st_full + 1;        // scores and dP of t are in registers (8 warp arrivals)
  uint64_t* p_full = st_free + 1;
  uint64_t* dv_done = p_full + 1;         // dV(t) has read P, and everything before it is done
  uint64_t* done = dv_done + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_t = (p.S + BT - 1) / BT;
  // The kv tile is the slowest grid index: CTAs are handed out in block-id order, so all the long tiles
  // (causal: small kt, up to 4x16 query tiles) start first and the short ones fill the tail.
  const int kt = blockIdx.z;  // kv tile
  const int kvh = blockIdx.x, b = blockIdx.y;
  const int group = p.H / p.Hkv;
  const int kv0 = kt * BT;
  const int row_base = b * p.S;
  const int qt_first = p.causal ? kt : 0;
  const int n_qt = n_t - qt_first;
  const int n_iter = group * n_qt;  // iteration t -> head kvh*group + t / n_qt, q tile qt_first + t % n_qt

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < Cfg::QS; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
    mbar_init(st_full, 1);
    mbar_init(p_full, 8);  // one arrival per softmax warp
    mbar_init(st_free, 8);
    mbar_init(dv_done, 1);
    mbar_init(done, 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) { prefetch_tmap(&tm_qkv); prefetch_tmap(&tm_do); }
  if (warp == 1) { tmem_alloc(tmem_holder, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_holder), 0);
  // S and dP are [query x kv] (TMEM lane = query row, as in the dQ kernel); their bf16 images P and dS
  // are stored [q rows][kv] and consumed as MN-major A operands (A^T) by the dV / dK products.
  const uint32_t tm_ST = tmem_base, tm_dPT = tmem_base + 128, tm_dK = tmem_base + 256, tm_dV = tmem_base + 256 + DH;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(kv_full, 2 * Cfg::T_BYTES);
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        tma_load_2d(sK + c * (BT * 128), &tm_qkv, kv_full, (p.H + kvh) * DH + c * 64, row_base + kv0);
        tma_load_2d(sV + c * (BT * 128), &tm_qkv, kv_full, (p.H + p.Hkv + kvh) * DH + c * 64, row_base + kv0);
      }
      int st = 0;
      uint32_t ph = 0;
      for (int t = 0; t < n_iter; ++t) {
        const int head = kvh * group + t / n_qt;
        const int qt = qt_first + t % n_qt;
        if (!mbar_wait(&q_empty[st], ph ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_arrive_expect_tx(&q_full[st], 2 * Cfg::T_BYTES);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          tma_load_2d(sQ + st * Cfg::T_BYTES + c * (BT * 128), &tm_qkv, &q_full[st], head * DH + c * 64,
                      row_base + qt * BT);
          tma_load_2d(sdO + st * Cfg::T_BYTES + c * (BT * 128), &tm_do, &q_full[st], head * DH + c * 64,
                      row_base + qt * BT);
        }
        if (++st == Cfg::QS) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = make_idesc_bf16(BT, BT, false, false);   // [q x kv], both K-major
    constexpr uint32_t idesc_g = make_idesc_bf16(BT, DH, true, true);     // [kv x dh] = A^T B, both MN-major
    const bool leader = elect_one();
    bool ok = mbar_wait_warp(kv_full, 0, p.status, ST_TIMEOUT_FULL);
    int st_s = 0;          // stage / phase of the next score issue
    uint32_t ph_s = 0;
    int st_g = 0;          // stage of the next gradient issue
    const uint64_t dK_ = make_smem_desc(smem_u32(sK), 16, 1024), dV_ = make_smem_desc(smem_u32(sV), 16, 1024);
    const uint64_t dPT = make_smem_desc(smem_u32(sPT), BT * 128, 1024);
    auto issue_scores = [&]() -> bool {
      if (!mbar_wait_warp(&q_full[st_s], ph_s, p.status, ST_TIMEOUT_FULL)) return false;
      tc_fence_after();
      const uint64_t dQ = make_smem_desc(smem_u32(sQ + st_s * Cfg::T_BYTES), 16, 1024);
      const uint64_t ddO = make_smem_desc(smem_u32(sdO + st_s * Cfg::T_BYTES), 16, 1024);
      if (leader) {
#pragma unroll
        for (int k = 0; k < DH / 16; ++k)
          umma_bf16_ss(tm_ST, smem_desc_at(dQ, k * 32), smem_desc_at(dK_, k * 32), idesc_s, k > 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < DH / 16; ++k)
          umma_bf16_ss(tm_dPT, smem_desc_at(ddO, k * 32), smem_desc_at(dV_, k * 32), idesc_s, k > 0 ? 1u : 0u);
        umma_commit(st_full);
      }
      __syncwarp();
      if (++st_s == Cfg::QS) { st_s = 0; ph_s ^= 1; }
      return true;
    };
    if (ok && n_iter > 0) ok = issue_scores();
    for (int t = 0; t < n_iter && ok; ++t) {
      if (t + 1 < n_iter) {
        if (!mbar_wait_warp(st_free, t & 1, p.status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        ok = issue_scores();
        if (!ok) break;
      }
      if (!mbar_wait_warp(p_full, t & 1, p.status, ST_TIMEOUT_MISC)) { ok = false; break; }
      tc_fence_after();
      const uint64_t ddS = make_smem_desc(smem_u32(sdST + (t & 1) * Cfg::PT_BYTES), BT * 128, 1024);
      const uint64_t dQ = make_smem_desc(smem_u32(sQ + st_g * Cfg::T_BYTES), BT * 128, 1024);
      const uint64_t ddO = make_smem_desc(smem_u32(sdO + st_g * Cfg::T_BYTES), BT * 128, 1024);
      if (leader) {
        if (p.spill_ds) {
          // the finished dS tile (bf16, [q rows][kv], scale included) also goes to global memory, where the dQ kernel
          // streams it back instead of recomputing scores. The bulk store reads shared memory asynchronously: the one of
          // t-1 must have been read out before dv_done(t), after which the softmax warps write that buffer again
          const int head = kvh * group + t / n_qt;
          const int qt = qt_first + t % n_qt;
          const uint8_t* src = sdST + (t & 1) * Cfg::PT_BYTES;
          tma_store_3d(&tm_ds, src, kv0, qt * BT, b * p.H + head);
          tma_store_3d(&tm_ds, src + BT * 128, kv0 + 64, qt * BT, b * p.H + head);
          tma_store_commit();
          tma_store_wait_read<1>();
        }
#pragma unroll
        for (int k = 0; k < BT / 16; ++k)   // k walks 16 query rows at a time in both operands
          umma_bf16_ss(tm_dV, smem_desc_at(dPT, k * (16 * 128)), smem_desc_at(ddO, k * (16 * 128)), idesc_g,
                       (t > 0 || k > 0) ? 1u : 0u);
        umma_commit(dv_done);
#pragma unroll
        for (int k = 0; k < BT / 16; ++k)
          umma_bf16_ss(tm_dK, smem_desc_at(ddS, k * (16 * 128)), smem_desc_at(dQ, k * (16 * 128)), idesc_g,
                       (t > 0 || k > 0) ? 1u : 0u);
        umma_commit(&q_empty[st_g]);
      }
      __syncwarp();
      if (++st_g == Cfg::QS) st_g = 0;
    }
    if (ok && leader) umma_commit(done);
    if (p.spill_ds && leader) tma_store_wait<0>();   // the stores are complete before the CTA retires
    __syncwarp();
  } else {
    const int sw = warp - 2;        // 0..7
    const int q = warp & 3;         // TMEM lane quarter
    const int half = sw >> 2;       // which 64 kv columns of the tile this warp handles
    const int r = q * 32 + lane;    // row inside the tile == TMEM lane (query row in the loop, kv row at the end)
    const int kv_idx = kv0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    bool ok = true;
    for (int t = 0; t < n_iter; ++t) {
      const int head = kvh * group + t / n_qt;
      const int qt = qt_first + t % n_qt;
      const int q0 = qt * BT;
      const int q_idx = q0 + r;
      const float2 sd = __ldg(p.stats + (static_cast<size_t>(b) * p.H + head) * p.S + min(q_idx, p.S - 1));
      uint8_t* dst_buf = sdST + (t & 1) * Cfg::PT_BYTES;
      // last visible kv column of this query row inside the tile (-1: row is past the sequence end)
      const bool diag = p.causal && qt == kt;
      int lim = min(diag ? r : BT - 1, p.S - 1 - kv0);
      if (q_idx >= p.S) lim = -1;
      const bool need_mask = diag || (q0 + BT > p.S) || (kv0 + BT > p.S);
      if (!mbar_wait_warp(st_full, t & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      // P = 2^(s * sl2 - lse2), dS = P * (dP * scale - delta * scale)
      uint32_t pv[64], dv[64];
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) tmem_ld_32x32(tm_ST + lane_off + (half * 2 + cc) * 32, pv + cc * 32);
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) tmem_ld_32x32(tm_dPT + lane_off + (half * 2 + cc) * 32, dv + cc * 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(st_free);
      const float neg_delta = -sd.y * p.scale;
#pragma unroll
      for (int i = 0; i < 64; i += 2) {
        fma2(pv[i], pv[i + 1], p.scale_log2, -sd.x);
        pv[i] = __float_as_uint(fast_exp2(__uint_as_float(pv[i])));
        pv[i + 1] = __float_as_uint(fast_exp2(__uint_as_float(pv[i + 1])));
        fma2(dv[i], dv[i + 1], p.scale, neg_delta);
      }
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (half * 64 + i > lim) pv[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 64; i += 2) {
        mul2(dv[i], dv[i + 1], __uint_as_float(pv[i]), __uint_as_float(pv[i + 1]));
        dv[i >> 1] = pack_bf16x2(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1]));
        pv[i >> 1] = pack_bf16x2(__uint_as_float(pv[i]), __uint_as_float(pv[i + 1]));
      }
      // dV(t-1) has read P; the dS buffer of this parity was let go of before
      if (t > 0 && !mbar_wait_warp(dv_done, (t - 1) & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        store_row32_sw128(sPT, r, half * 2 + cc, pv + cc * 16);
        store_row32_sw128(dst_buf, r, half * 2 + cc, dv + cc * 16);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok && mbar_wait_warp(done, 0, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      constexpr int CPW = DH / 64;  // 32-column chunks per warp and matrix
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t src = which == 0 ? tm_dK : tm_dV;
        const int col0 = (which == 0 ? (p.H + kvh) : (p.H + p.Hkv + kvh)) * DH;
#pragma unroll 1
        for (int cc = 0; cc < CPW; ++cc) {
          const int c = half * CPW + cc;
          uint32_t v[32];
          tmem_ld_32x32(src + lane_off + c * 32, v);
          tmem_ld_wait();
          if (kv_idx < p.S) {
            __nv_bfloat16* dst = p.dqkv + static_cast<size_t>(row_base + kv_idx) * p.ld_dqkv + col0 + c * 32;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
              w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
              w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
              w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
              *reinterpret_cast<uint4*>(dst + u * 8) = w;
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

// Pipeline at head dimension 128: scores and dP have barriers of their own, so the exponentials of iteration t+1 (which need
// the scores only) run under the gradient products of iteration t, and dS follows when dP arrives. Order of the tensor work:
//   S(t+1) | dV(t) += P(t)^T dO(t) | dK(t) += dS(t)^T Q(t) | dP(t+1)
// S(t+1) needs Q(t+1), so Q has two stages; dO(t) is free after dV(t), two products before dP(t+1) needs its successor,
// so one stage is enough where shared memory holds seven 32 KB tiles (K, V, 2 Q, dO, P, dS).
// P is single: dV(t) has read it (dv_done) long before the exponentials of t+1 are stored. Until then the two score
// products of an iteration were one group, which the softmax warps waited for as a whole, and at 128 the loads,
// the scores, the softmax and the gradient products of an iteration ran one after another: 2 x 2048 tokens of 32 heads,
// causal, 241 us then and 176 us so. One thread issues here: a whole warp walking through the loop, which the kernel above gains
// from, is level at 2 x 2048 tokens and loses 5 % at 1 x 2048.
struct DkvSplitCfg {
  static constexpr int DH = 128;
  static constexpr int QS = 2;                        // Q stages; dO, P and dS have one
  static constexpr int T_BYTES = BT * DH * 2;         // one [128 x DH] tile
  static constexpr int PT_BYTES = BT * BT * 2;
  static constexpr int TILE_BYTES = (2 + QS + 1) * T_BYTES + 2 * PT_BYTES;
  static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = 512;  // S 128 | dP 128 | dK DH | dV DH
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
};

__global__ void __launch_bounds__(BWD_THREADS, 1)
attention_bwd_dkv_split_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                               const __grid_constant__ CUtensorMap tm_ds, const BwdParams p) {
  using Cfg = DkvSplitCfg;
  constexpr int DH = Cfg::DH, NCH = DH / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::T_BYTES;
  uint8_t* sQ = sV + Cfg::T_BYTES;                 // QS stages
  uint8_t* sdO = sQ + Cfg::QS * Cfg::T_BYTES;
  uint8_t* sPT = sdO + Cfg::T_BYTES;
  uint8_t* sdST = sPT + Cfg::PT_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sdST + Cfg::PT_BYTES);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;             // QS
  uint64_t* q_empty = q_full + Cfg::QS;    // QS
  uint64_t* do_full = q_empty + Cfg::QS;
  uint64_t* do_empty = do_full + 1;
  uint64_t* s_full = do_empty + 1;         // scores of t are in tensor memory
  uint64_t* dp_full = s_full + 1;          // dP of t is; every earlier product has completed and dS may be rewritten
  uint64_t* p_full = dp_full + 1;          // P of t is in shared memory (8 warp arrivals), the scores have been read
  uint64_t* ds_full = p_full + 1;          // dS of t is, dP has been read
  uint64_t* dv_done = ds_full + 1;         // dV(t) has read P
  uint64_t* done = dv_done + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_t = (p.S + BT - 1) / BT;
  // The kv tile is the slowest grid index: CTAs are handed out in block-id order, so all the long tiles
  // (causal: small kt, up to 4x16 query tiles) start first and the short ones fill the tail.
  const int kt = blockIdx.z;  // kv tile
  const int kvh = blockIdx.x, b = blockIdx.y;
  const int group = p.H / p.Hkv;
  const int kv0 = kt * BT;
  const int row_base = b * p.S;
  const int qt_first = p.causal ? kt : 0;
  const int n_qt = n_t - qt_first;
  const int n_iter = group * n_qt;  // iteration t -> head kvh*group + t / n_qt, q tile qt_first + t % n_qt

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < Cfg::QS; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);  // one arrival per softmax warp
    mbar_init(ds_full, 8);
    mbar_init(dv_done, 1);
    mbar_init(done, 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) { prefetch_tmap(&tm_qkv); prefetch_tmap(&tm_do); }
  if (warp == 1) { tmem_alloc(tmem_holder, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_holder);
  // S and dP are [query x kv] (TMEM lane = query row, as in the dQ kernel); their bf16 images P and dS
  // are stored [q rows][kv] and consumed as MN-major A operands (A^T) by the dV / dK products.
  const uint32_t tm_ST = tmem_base, tm_dPT = tmem_base + 128, tm_dK = tmem_base + 256, tm_dV = tmem_base + 256 + DH;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(kv_full, 2 * Cfg::T_BYTES);
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        tma_load_2d(sK + c * (BT * 128), &tm_qkv, kv_full, (p.H + kvh) * DH + c * 64, row_base + kv0);
        tma_load_2d(sV + c * (BT * 128), &tm_qkv, kv_full, (p.H + p.Hkv + kvh) * DH + c * 64, row_base + kv0);
      }
      int qs = 0;
      uint32_t qph = 0;
      for (int t = 0; t < n_iter; ++t) {
        const int head = kvh * group + t / n_qt;
        const int qt = qt_first + t % n_qt;
        if (!mbar_wait(&q_empty[qs], qph ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_arrive_expect_tx(&q_full[qs], Cfg::T_BYTES);
#pragma unroll
        for (int c = 0; c < NCH; ++c)
          tma_load_2d(sQ + qs * Cfg::T_BYTES + c * (BT * 128), &tm_qkv, &q_full[qs], head * DH + c * 64,
                      row_base + qt * BT);
        if (++qs == Cfg::QS) { qs = 0; qph ^= 1; }
        if (!mbar_wait(do_empty, (t & 1) ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_arrive_expect_tx(do_full, Cfg::T_BYTES);
#pragma unroll
        for (int c = 0; c < NCH; ++c)
          tma_load_2d(sdO + c * (BT * 128), &tm_do, do_full, head * DH + c * 64, row_base + qt * BT);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BT, BT, false, false);   // [q x kv], both K-major
      constexpr uint32_t idesc_g = make_idesc_bf16(BT, DH, true, true);     // [kv x dh] = A^T B, both MN-major
      bool ok = mbar_wait(kv_full, 0, p.status, ST_TIMEOUT_FULL);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), adO = smem_u32(sdO), aPT = smem_u32(sPT), adS = smem_u32(sdST);
      int qn = 0;                    // Q stage and phase of the next score product
      uint32_t qn_ph = 0;
      int qg = 0;                    // Q stage of the next dK product
      // D = A B^T over DH, both K-major
      auto score_product = [&](uint32_t d, uint32_t a, uint32_t b) {
#pragma unroll
        for (int k = 0; k < DH / 16; ++k) {
          const uint32_t off = (k >> 2) * (BT * 128) + (k & 3) * 32;
          umma_bf16_ss(d, make_smem_desc(a + off, 16, 1024), make_smem_desc(b + off, 16, 1024), idesc_s, k > 0 ? 1u : 0u);
        }
      };
      // D += A^T B over the 128 query rows, 16 at a time in both operands
      auto grad_product = [&](uint32_t d, uint32_t a, uint32_t b, bool acc) {
#pragma unroll
        for (int k = 0; k < BT / 16; ++k)
          umma_bf16_ss(d, make_smem_desc(a + k * (16 * 128), BT * 128, 1024),
                       make_smem_desc(b + k * (16 * 128), BT * 128, 1024), idesc_g, (acc || k > 0) ? 1u : 0u);
      };
      auto issue_s = [&]() -> bool {
        if (!mbar_wait(&q_full[qn], qn_ph, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        score_product(tm_ST, smem_u32(sQ + qn * Cfg::T_BYTES), aK);
        umma_commit(s_full);
        if (++qn == Cfg::QS) { qn = 0; qn_ph ^= 1; }
        return true;
      };
      auto issue_dp = [&](int t) -> bool {
        if (!mbar_wait(do_full, t & 1, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        // dp_full lets the softmax warps write dS again: its last bulk store must have been read out
        if (p.spill_ds) tma_store_wait_read<0>();
        score_product(tm_dPT, adO, aV);
        umma_commit(dp_full);
        return true;
      };
      if (n_iter > 0) ok = ok && issue_s() && issue_dp(0);
      for (int t = 0; t < n_iter && ok; ++t) {
        const bool more = t + 1 < n_iter;
        if (!mbar_wait(p_full, t & 1, p.status, ST_TIMEOUT_MISC)) { ok = false; break; }
        tc_fence_after();
        if (more && !issue_s()) { ok = false; break; }
        grad_product(tm_dV, aPT, adO, t > 0);
        umma_commit(dv_done);
        umma_commit(do_empty);
        if (!mbar_wait(ds_full, t & 1, p.status, ST_TIMEOUT_MISC)) { ok = false; break; }
        tc_fence_after();
        if (p.spill_ds) {
          // the finished dS tile (bf16, [q rows][kv], scale included) also goes to global memory, where
          // the dQ kernel streams it back instead of recomputing scores
          const int head = kvh * group + t / n_qt;
          const int qt = qt_first + t % n_qt;
          tma_store_3d(&tm_ds, sdST, kv0, qt * BT, b * p.H + head);
          tma_store_3d(&tm_ds, sdST + BT * 128, kv0 + 64, qt * BT, b * p.H + head);
          tma_store_commit();
        }
        grad_product(tm_dK, adS, smem_u32(sQ + qg * Cfg::T_BYTES), t > 0);
        umma_commit(&q_empty[qg]);
        if (++qg == Cfg::QS) qg = 0;
        if (more && !issue_dp(t + 1)) { ok = false; break; }
      }
      if (ok) umma_commit(done);
      if (p.spill_ds) tma_store_wait<0>();   // the stores are complete before the CTA retires
    }
  } else {
    const int sw = warp - 2;        // 0..7
    const int q = warp & 3;         // TMEM lane quarter
    const int half = sw >> 2;       // which 64 kv columns of the tile this warp handles
    const int r = q * 32 + lane;    // row inside the tile == TMEM lane (query row in the loop, kv row at the end)
    const int kv_idx = kv0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    bool ok = true;
    for (int t = 0; t < n_iter; ++t) {
      const int head = kvh * group + t / n_qt;
      const int qt = qt_first + t % n_qt;
      const int q0 = qt * BT;
      const int q_idx = q0 + r;
      const float2 sd = __ldg(p.stats + (static_cast<size_t>(b) * p.H + head) * p.S + min(q_idx, p.S - 1));
      // last visible kv column of this query row inside the tile (-1: row is past the sequence end)
      const bool diag = p.causal && qt == kt;
      int lim = min(diag ? r : BT - 1, p.S - 1 - kv0);
      if (q_idx >= p.S) lim = -1;
      const bool need_mask = diag || (q0 + BT > p.S) || (kv0 + BT > p.S);
      if (!mbar_wait_warp(s_full, t & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      // P = 2^(s * sl2 - lse2), kept in fp32 registers for dS
      uint32_t pv[64];
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) tmem_ld_32x32(tm_ST + lane_off + (half * 2 + cc) * 32, pv + cc * 32);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 64; i += 2) {
        fma2(pv[i], pv[i + 1], p.scale_log2, -sd.x);
        pv[i] = __float_as_uint(fast_exp2(__uint_as_float(pv[i])));
        pv[i + 1] = __float_as_uint(fast_exp2(__uint_as_float(pv[i + 1])));
      }
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (half * 64 + i > lim) pv[i] = 0u;
      }
      if (t > 0 && !mbar_wait_warp(dv_done, (t - 1) & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          pk[i >> 1] = pack_bf16x2(__uint_as_float(pv[cc * 32 + i]), __uint_as_float(pv[cc * 32 + i + 1]));
        store_row32_sw128(sPT, r, half * 2 + cc, pk);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      // dS = P * (dP * scale - delta * scale)
      if (!mbar_wait_warp(dp_full, t & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const float neg_delta = -sd.y * p.scale;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t dv[32], dk[16];
        tmem_ld_32x32(tm_dPT + lane_off + (half * 2 + cc) * 32, dv);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          fma2(dv[i], dv[i + 1], p.scale, neg_delta);
          mul2(dv[i], dv[i + 1], __uint_as_float(pv[cc * 32 + i]), __uint_as_float(pv[cc * 32 + i + 1]));
          dk[i >> 1] = pack_bf16x2(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1]));
        }
        store_row32_sw128(sdST, r, half * 2 + cc, dk);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (ok && mbar_wait_warp(done, 0, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      constexpr int CPW = DH / 64;  // 32-column chunks per warp and matrix
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t src = which == 0 ? tm_dK : tm_dV;
        const int col0 = (which == 0 ? (p.H + kvh) : (p.H + p.Hkv + kvh)) * DH;
#pragma unroll 1
        for (int cc = 0; cc < CPW; ++cc) {
          const int c = half * CPW + cc;
          uint32_t v[32];
          tmem_ld_32x32(src + lane_off + c * 32, v);
          tmem_ld_wait();
          if (kv_idx < p.S) {
            __nv_bfloat16* dst = p.dqkv + static_cast<size_t>(row_base + kv_idx) * p.ld_dqkv + col0 + c * 32;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
              w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
              w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
              w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
              *reinterpret_cast<uint4*>(dst + u * 8) = w;
            }
          }
          __syncwarp();   // rows past the end have skipped the stores; the next tensor-memory load needs the whole warp
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

// --------------------------------------------------------------------------- dQ
template <int DH>
struct DqCfg {
  static constexpr bool PDB = (DH == 64);        // double-buffer dS
  static constexpr int NPB = PDB ? 2 : 1;
  static constexpr int KS = (DH == 64) ? 2 : 1;  // (K, V) ring stages
  static constexpr int T_BYTES = BT * DH * 2;
  static constexpr int DS_BYTES = BT * BT * 2;
  static constexpr int TILE_BYTES = 2 * T_BYTES + KS * 2 * T_BYTES + NPB * DS_BYTES;
  static constexpr int SMEM_BYTES = TILE_BYTES + 1024 + 128;
  static constexpr int TMEM_COLS = 512;  // S 128 | dP 128 | dQ DH
};

template <int DH>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attention_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                        const BwdParams p) {
  using Cfg = DqCfg<DH>;
  constexpr int NCH = DH / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + Cfg::T_BYTES;
  uint8_t* sK = sdO + Cfg::T_BYTES;               // KS stages
  uint8_t* sV = sK + Cfg::KS * Cfg::T_BYTES;      // KS stages
  uint8_t* sdS = sV + Cfg::KS * Cfg::T_BYTES;     // NPB buffers
  uint64_t* bars = reinterpret_cast<uint64_t*>(sdS + Cfg::NPB * Cfg::DS_BYTES);
  uint64_t* q_full = bars;
  uint64_t* kv_full = bars + 1;            // KS
  uint64_t* kv_empty = kv_full + Cfg::KS;  // KS
  uint64_t* s_full = kv_empty + Cfg::KS;
  uint64_t* p_full = s_full + 1;
  uint64_t* done = p_full + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_t = (p.S + BT - 1) / BT;
  const int qt = n_t - 1 - blockIdx.z;   // slowest grid index: longest rows of tiles first over the whole grid
  const int head = blockIdx.x, b = blockIdx.y;
  const int kvh = head / (p.H / p.Hkv);
  const int q0 = qt * BT;
  const int row_base = b * p.S;
  const int n_blocks = p.causal ? (qt + 1) : n_t;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < Cfg::KS; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(done, 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) { prefetch_tmap(&tm_qkv); prefetch_tmap(&tm_do); }
  if (warp == 1) { tmem_alloc(tmem_holder, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_holder);
  const uint32_t tm_S = tmem_base, tm_dP = tmem_base + 128, tm_dQ = tmem_base + 256;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, 2 * Cfg::T_BYTES);
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        tma_load_2d(sQ + c * (BT * 128), &tm_qkv, q_full, head * DH + c * 64, row_base + q0);
        tma_load_2d(sdO + c * (BT * 128), &tm_do, q_full, head * DH + c * 64, row_base + q0);
      }
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_blocks; ++j) {
        if (!mbar_wait(&kv_empty[st], ph ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_arrive_expect_tx(&kv_full[st], 2 * Cfg::T_BYTES);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          tma_load_2d(sK + st * Cfg::T_BYTES + c * (BT * 128), &tm_qkv, &kv_full[st], (p.H + kvh) * DH + c * 64,
                      row_base + j * BT);
          tma_load_2d(sV + st * Cfg::T_BYTES + c * (BT * 128), &tm_qkv, &kv_full[st],
                      (p.H + p.Hkv + kvh) * DH + c * 64, row_base + j * BT);
        }
        if (++st == Cfg::KS) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BT, BT, false, false);
      constexpr uint32_t idesc_g = make_idesc_bf16(BT, DH, false, true);
      bool ok = mbar_wait(q_full, 0, p.status, ST_TIMEOUT_FULL);
      int st_s = 0, st_g = 0;
      uint32_t ph_s = 0;
      const uint32_t aQ = smem_u32(sQ), adO = smem_u32(sdO);
      auto issue_scores = [&]() -> bool {
        if (!mbar_wait(&kv_full[st_s], ph_s, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        const uint32_t bK = smem_u32(sK + st_s * Cfg::T_BYTES), bV = smem_u32(sV + st_s * Cfg::T_BYTES);
#pragma unroll
        for (int k = 0; k < DH / 16; ++k) {
          const uint32_t off = (k >> 2) * (BT * 128) + (k & 3) * 32;
          umma_bf16_ss(tm_S, make_smem_desc(aQ + off, 16, 1024), make_smem_desc(bK + off, 16, 1024), idesc_s,
                       k > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int k = 0; k < DH / 16; ++k) {
          const uint32_t off = (k >> 2) * (BT * 128) + (k & 3) * 32;
          umma_bf16_ss(tm_dP, make_smem_desc(adO + off, 16, 1024), make_smem_desc(bV + off, 16, 1024), idesc_s,
                       k > 0 ? 1u : 0u);
        }
        umma_commit(s_full);
        if (++st_s == Cfg::KS) { st_s = 0; ph_s ^= 1; }
        return true;
      };
      auto issue_grad = [&](int j) {
        const int pb = Cfg::PDB ? (j & 1) : 0;
        const uint32_t adS = smem_u32(sdS + pb * Cfg::DS_BYTES), bK = smem_u32(sK + st_g * Cfg::T_BYTES);
#pragma unroll
        for (int k = 0; k < BT / 16; ++k) {
          const uint32_t aoff = (k >> 2) * (BT * 128) + (k & 3) * 32;
          umma_bf16_ss(tm_dQ, make_smem_desc(adS + aoff, 16, 1024),
                       make_smem_desc(bK + k * (16 * 128), BT * 128, 1024), idesc_g, (j > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&kv_empty[st_g]);
        if (++st_g == Cfg::KS) st_g = 0;
      };
      if (ok) ok = issue_scores();
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (!mbar_wait(p_full, j & 1, p.status, ST_TIMEOUT_MISC)) { ok = false; break; }
        tc_fence_after();
        if (Cfg::PDB) {
          if (j + 1 < n_blocks) ok = issue_scores();
          issue_grad(j);
        } else {
          issue_grad(j);
          if (j + 1 < n_blocks) ok = issue_scores();
        }
      }
      if (ok) umma_commit(done);
    }
  } else {
    const int sw = warp - 2;
    const int q = warp & 3;
    const int half = sw >> 2;
    const int r = q * 32 + lane;
    const int q_idx = q0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    float lse2 = 0.f, del = 0.f;
    if (q_idx < p.S) {
      const float2 sd = p.stats[(static_cast<size_t>(b) * p.H + head) * p.S + q_idx];
      lse2 = sd.x;
      del = sd.y;
    }
    bool ok = true;
    for (int j = 0; j < n_blocks; ++j) {
      if (!mbar_wait_warp(s_full, j & 1, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int kv0 = j * BT;
      const bool diag = p.causal && j == n_blocks - 1;
      const bool need_mask = diag || (kv0 + BT > p.S) || (q0 + BT > p.S);
      int lim = min(diag ? r : BT - 1, p.S - 1 - kv0);
      if (q_idx >= p.S) lim = -1;
      uint8_t* ds_buf = sdS + (Cfg::PDB ? (j & 1) : 0) * Cfg::DS_BYTES;
      if (need_mask) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
          bwd_chunk<true>(tm_S, tm_dP, lane_off, half * 2 + cc, r, lim, p.scale_log2, lse2, del * p.scale,
                                 p.scale, ds_buf);
      } else {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc)
          bwd_chunk<false>(tm_S, tm_dP, lane_off, half * 2 + cc, r, lim, p.scale_log2, lse2, del * p.scale,
                                  p.scale, ds_buf);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok && mbar_wait_warp(done, 0, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      constexpr int CPW = DH / 64;
#pragma unroll 1
      for (int cc = 0; cc < CPW; ++cc) {
        const int c = half * CPW + cc;
        uint32_t v[32];
        tmem_ld_32x32(tm_dQ + lane_off + c * 32, v);
        tmem_ld_wait();
        if (q_idx < p.S) {
          __nv_bfloat16* dst = p.dqkv + static_cast<size_t>(row_base + q_idx) * p.ld_dqkv + head * DH + c * 32;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
            *reinterpret_cast<uint4*>(dst + u * 8) = w;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}


// --------------------------------------------------------------------------- dQ from stored dS
// When the dK/dV kernel has spilled its dS tiles (bf16 [B*H, S, S], scale included), dQ = dS K is a
// plain streamed product: no scores, no exponentials. One CTA per (query tile, head, batch) walks the
// kv tiles in ascending order through a TMA ring of (dS tile, K tile) pairs and accumulates in TMEM.
// It is bound by the bytes of dS (half of S x S per head under the causal mask). A CTA's stream is short (16 tiles at 2048
// tokens), so its start and its epilogue count: a stage holds half a kv tile, and two CTAs share an SM, one streaming while
// the other starts or ends (8 x 2048 tokens of 16 heads of 64,
// the whole backward 398 us with one CTA of twice the stages, 384 so).
template <int DH>
struct DqsCfg {
  static constexpr int KT = BT / 2;                      // kv rows per stage
  static constexpr int DS_BYTES = BT * KT * 2;
  static constexpr int K_BYTES = KT * DH * 2;
  static constexpr int STAGE_BYTES = DS_BYTES + K_BYTES;
  static constexpr int STAGES = (DH == 64) ? 4 : 3;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 128;
  static constexpr int TMEM_COLS = DH;
  static_assert(2 * (SMEM_BYTES + 1024) <= 227 * 1024, "two CTAs per SM");
};

template <int DH>
__global__ void __launch_bounds__(BWD_THREADS, 2)
attention_bwd_dq_stream_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_ds,
                               const BwdParams p) {
  using Cfg = DqsCfg<DH>;
  constexpr int NCH = DH / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + Cfg::STAGES;
  uint64_t* done = empty + Cfg::STAGES;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_t = (p.S + BT - 1) / BT;
  const int qt = n_t - 1 - blockIdx.z;   // slowest grid index: longest rows of tiles first over the whole grid
  const int head = blockIdx.x, b = blockIdx.y;
  const int kvh = head / (p.H / p.Hkv);
  const int q0 = qt * BT;
  const int row_base = b * p.S;
  const int n_blocks = 2 * (p.causal ? (qt + 1) : n_t);    // half tiles

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) { prefetch_tmap(&tm_k); prefetch_tmap(&tm_ds); }
  if (warp == 1) { tmem_alloc(tmem_holder, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm_dQ = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_holder), 0);

  if (warp == 0) {
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_blocks; ++j) {
        if (!mbar_wait(&empty[st], ph ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
        uint8_t* sdS = smem + st * Cfg::STAGE_BYTES;
        uint8_t* sK = sdS + Cfg::DS_BYTES;
        mbar_arrive_expect_tx(&full[st], Cfg::STAGE_BYTES);
        tma_load_3d(sdS, &tm_ds, &full[st], j * Cfg::KT, q0, b * p.H + head);
#pragma unroll
        for (int c = 0; c < NCH; ++c)
          tma_load_2d(sK + c * (Cfg::KT * 128), &tm_k, &full[st], (p.H + kvh) * DH + c * 64, row_base + j * Cfg::KT);
        if (++st == Cfg::STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_g = make_idesc_bf16(BT, DH, false, true);
    const bool leader = elect_one();
    int st = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int j = 0; j < n_blocks && ok; ++j) {
      ok = mbar_wait_warp(&full[st], ph, p.status, ST_TIMEOUT_FULL);
      if (!ok) break;
      tc_fence_after();
      const uint64_t da = make_smem_desc(smem_u32(smem + st * Cfg::STAGE_BYTES), 16, 1024);
      const uint64_t db = make_smem_desc(smem_u32(smem + st * Cfg::STAGE_BYTES + Cfg::DS_BYTES), Cfg::KT * 128, 1024);
      if (leader) {
#pragma unroll
        for (int k = 0; k < Cfg::KT / 16; ++k)
          umma_bf16_ss(tm_dQ, smem_desc_at(da, k * 32), smem_desc_at(db, k * (16 * 128)), idesc_g, (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[st]);
      }
      __syncwarp();
      if (++st == Cfg::STAGES) { st = 0; ph ^= 1; }
    }
    if (ok && leader) umma_commit(done);
    __syncwarp();
  } else {
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r = q * 32 + lane;
    const int q_idx = q0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    if (mbar_wait_warp(done, 0, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      constexpr int CPW = DH / 64;
#pragma unroll 1
      for (int cc = 0; cc < CPW; ++cc) {
        const int c = half * CPW + cc;
        uint32_t v[32];
        tmem_ld_32x32(tm_dQ + lane_off + c * 32, v);
        tmem_ld_wait();
        if (q_idx < p.S) {
          __nv_bfloat16* dst = p.dqkv + static_cast<size_t>(row_base + q_idx) * p.ld_dqkv + head * DH + c * 32;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
            *reinterpret_cast<uint4*>(dst + u * 8) = w;
          }
        }
        __syncwarp();   // rows past the end have skipped the stores; the next tensor-memory load needs the whole warp
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tm_dQ, Cfg::TMEM_COLS);
}

template <int DH>
static int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& td, const CUtensorMap& tds, const BwdParams& p,
                      cudaStream_t stream) {
  constexpr int DKV_SMEM = DH == 64 ? DkvCfg::SMEM_BYTES : DkvSplitCfg::SMEM_BYTES;
  auto k1 = DH == 64 ? attention_bwd_dkv_kernel : attention_bwd_dkv_split_kernel;
  auto k2 = attention_bwd_dq_kernel<DH>;
  auto k3 = attention_bwd_dq_stream_kernel<DH>;
  static PerDeviceOnce a1, a2, a3;
  if (allow_smem(a1, k1, DKV_SMEM, SB_ERR_LAUNCH) || allow_smem(a2, k2, DqCfg<DH>::SMEM_BYTES, SB_ERR_LAUNCH) ||
      allow_smem(a3, k3, DqsCfg<DH>::SMEM_BYTES, SB_ERR_LAUNCH))
    return SB_ERR_LAUNCH;
  const int n_t = (p.S + BT - 1) / BT;
  k1<<<dim3(p.Hkv, p.B, n_t), BWD_THREADS, DKV_SMEM, stream>>>(tq, td, tds, p);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  if (p.spill_ds) k3<<<dim3(p.H, p.B, n_t), BWD_THREADS, DqsCfg<DH>::SMEM_BYTES, stream>>>(tk, tds, p);
  else k2<<<dim3(p.H, p.B, n_t), BWD_THREADS, DqCfg<DH>::SMEM_BYTES, stream>>>(tq, td, p);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

}  // namespace sb

using namespace sb;

// qkv, dqkv: bf16 [B*S, ld]; O, dO: bf16 [B*S, ld_o / ld_do] (H*dh columns); lse: fp32 [B,H,S];
// delta: scratch of 2*B*H*S floats written here ((lse*log2e, delta) pairs). dqkv receives dQ | dK | dV in
// the qkv layout. ds_scratch (optional): B*H*S*round_up(S, 64) bf16; with it the dK/dV kernel stores its
// dS tiles there and dQ is computed by streaming them back (faster: no second pass over the scores);
// without it dQ recomputes scores and exponentials.
extern "C" size_t sb_attention_bwd_ds_elems(int B, int S, int H) {
  return static_cast<size_t>(B) * H * S * ((S + 63) / 64 * 64);
}

extern "C" int sb_attention_bwd(const void* qkv, const void* O, const float* lse, const void* dO, void* dqkv,
                                float* delta, void* ds_scratch, int B, int S, int H, int Hkv, int dh, int ld,
                                int ld_o, int ld_do, float scale, int causal, int* status, void* stream_) {
  if (B <= 0 || S <= 0 || H <= 0 || Hkv <= 0 || (H % Hkv) || (dh != 64 && dh != 128)) return SB_ERR_ARG;
  if (B > 65535 || (S + 127) / 128 > 65535) return SB_ERR_TOO_LARGE;   // grid y / z limits
  if ((ld & 7) || (reinterpret_cast<uintptr_t>(dqkv) & 15)) return SB_ERR_ALIGN;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  CUtensorMap tq, tk, td;
  int rc = make_tmap_2d_bf16(&tq, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(B) * S, ld, 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tk, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(B) * S, ld, 64, BT / 2);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&td, dO, static_cast<uint64_t>(H) * dh, static_cast<uint64_t>(B) * S, ld_do, 64, 128);
  if (rc) return rc;
  if ((ld_o & 7) || (ld_do & 7) || (reinterpret_cast<uintptr_t>(O) & 15) || (reinterpret_cast<uintptr_t>(dO) & 15))
    return SB_ERR_ALIGN;
  attn_delta_kernel<<<dim3((B * S + DL_ROWS - 1) / DL_ROWS, (H * dh + DL_COLS - 1) / DL_COLS), DL_ROWS * 32, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(O), static_cast<const __nv_bfloat16*>(dO), lse, reinterpret_cast<float2*>(delta), B * S, S, H,
      dh, ld_o, ld_do);
  if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  BwdParams p;
  p.B = B; p.S = S; p.H = H; p.Hkv = Hkv;
  p.ld_dqkv = ld;
  p.scale = scale;
  p.scale_log2 = scale * LOG2E;
  p.causal = causal;
  p.lse = lse;
  p.stats = reinterpret_cast<const float2*>(delta);
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.status = status;
  p.spill_ds = ds_scratch ? 1 : 0;
  CUtensorMap tds = tq;   // placeholder when unused
  if (ds_scratch) {
    const uint64_t sp = (static_cast<uint64_t>(S) + 63) / 64 * 64;
    rc = make_tmap_3d_bf16(&tds, ds_scratch, S, S, static_cast<uint64_t>(B) * H, sp, sp * S, 64, 128);
    if (rc) return rc;
  }
  return dh == 64 ? launch_bwd<64>(tq, tk, td, tds, p, stream) : launch_bwd<128>(tq, tk, td, tds, p, stream);
}
