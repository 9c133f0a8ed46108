// GQA flash-attention forward for sm_100a, head dimensions 64 and 128, two query tiles per CTA.
//
// One CTA owns 256 query rows of one (head, batch) as two 128-row tiles. Each tile has its own
// output accumulator O_t in tensor memory and its own group of four softmax warps, so while the warps of one tile run their exponentials the tensor cores work on
// the other tile's products. The output accumulator stays in tensor memory for the whole loop:
// P V is accumulated there by the MMA itself, and a row is rescaled when its running maximum has grown
// since the reference point used in the exponent: at head dimension 64 by more than 2^8 (bf16 P then
// stays below 2^8, far inside its range), which on real score distributions happens in the first blocks
// only; at 128 by anything. There the reference is the running maximum itself, as in the one-tile kernel,
// so the largest weight of a row is 1 and has no rounding; with the 2^8 margin the error against float64
// was 2 % larger for unit scores and 20 % larger for scores of twice the spread. The rescales cost 5 %. The row sum uses
// the same reference point, so the final O / l and the log-sum-exp are exact regardless of when a rescale happened.
//
// Same interface, layout and semantics as the one-tile kernel (attention_fwd_tcgen05.cu): fused
// activation matrix qkv [B*S, ld] = [q heads | k heads | v heads], scores scaled by 1/sqrt(dh),
// causal mask j > i, fp32 softmax, bf16 P, O [B*S, H*dh] bf16, LSE [B, H, S] fp32. KV blocks are
// visited in ascending order and every decision depends on the data only, so results are bitwise
// repeatable. Counterpart in the reference: the per-(sequence, head) GEMM + scale_mask + softmax
// chain of scirust-sciagent/src/cuda_model.rs:796-832.
//
// A softmax thread holds its whole 128-column score row in registers (one pass over tensor memory),
// scales it with packed fp32 pairs (fma.rn.f32x2, add.rn.f32x2: half the issue slots of scalar
// code) and takes the row maximum with three-input max. What bounds the kernel is the chain inside a tile (scores, maximum, rescale,
// exponentials, P, P V) and, in a long run, the power cap: 5000 tokens of 32 heads of 128 run at 1.96 GHz for a few
// milliseconds and at 1.75 after that. Two softmax warps share a scheduler, so the special-function unit needs 2048 cycles for a
// block of both tiles, and so does the tensor pipe at head dimension 128; a block takes about 3300 (2800 at 64; 3500 with P in
// shared memory; profiles/attention_issue_and_softmax.md).
//  - P goes to tensor memory, from where the tensor core takes it as its A operand. A product with both operands in shared memory reads
//    8 KB in the 64 cycles that it runs, all that shared memory gives; with P there too, its stores, the products and the tiles
//    that arrive asked shared memory for 3000 cycles a block. Its two halves of 64 columns are handed over one by one.
//  - At head dimension 128 tensor memory is full with one score accumulator (128 columns), P (2 x 64) and O (2 x 128): the tiles take
//    turns with the accumulator, which is free again when a tile has its scores in registers, and so run half a block
//    apart, one in its exponentials while the other waits, loads and rescales. At 64 each has its own.
//  - One warp issues for both tiles in the order S0(j) PV0(j-1) S1(j) PV1(j-1), in which they come up: the scores of a block are there
//    when the block before is done.
//  - The issuing warp walks through its loop as a whole and one lane issues: descriptors and addresses stay in uniform
//    registers. As the loop of a single thread a product cost it 70 to 150 cycles to issue, more than to run.
//  - The mask is applied to the scores of the blocks that need one; as a select beside every exponential it
//    cost all blocks a third of their instructions.
// The softmax warpgroups take the registers that the issuing one does not need (setmaxnreg), so rows stay unspilled.
// us with P in shared memory and an issuing warp per tile / now, causal, calls back to back on one input, 32 heads of 128: 5000 tokens
// 211 / 198 (1033 TFLOP/s; in a long run on new inputs 238 / 224), 4096 146 / 134, 2 x 2048 93 / 85; 16 heads of 64: 8 x 2048 140 / 128,
// 2 x 2048 40.5 / 37.4; the same bits. Measured and dropped: the rescale in four warps of its own (5000 tokens 222: the softmax
// warps wait longer for one another than for the rescale), two warps a row (212), exponentials of the tiles in strict turns (level).
//
// Warps: 0 TMA producer, 1 MMA issuer, 2 and 3 idle, 4-7 softmax of tile 0, 8-11 softmax of tile 1.
#include "sm100_ptx.cuh"
#include "api.h"
#include "per_device.h"

namespace sb {

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

namespace attpp {

constexpr int BM = 128;        // query rows per tile
constexpr int BN = 128;        // kv rows per block
constexpr int THREADS = 384;
// Registers a thread: 168 at launch for all three warpgroups, shared out as 56 (producer, issuer) + 2 x 224 (softmax).
constexpr int REGS_ISSUE = 56, REGS_SOFTMAX = 224;
static_assert(REGS_ISSUE + 2 * REGS_SOFTMAX <= 3 * 168, "the shares draw on the registers of the launch");
constexpr int HALF = BN / 2;   // columns of P that are handed over at once
constexpr int TMEM_COLS = 512;

template <int DH>
struct Cfg {
  static constexpr int NCH = DH / 64;                  // 64-column chunks per head
  static constexpr int KS = 3;                         // K ring stages
  static constexpr int VS = DH == 64 ? 3 : 2;          // V ring stages
  static constexpr int Q_BYTES = BM * DH * 2;
  static constexpr int KV_BYTES = BN * DH * 2;
  static constexpr int TILE_BYTES = 2 * Q_BYTES + (KS + VS) * KV_BYTES;
  static constexpr int SMEM_BYTES = TILE_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
  // tensor memory: score accumulators (one that the tiles take turns with at 128, one each at 64), P as bf16 pairs, O
  static constexpr int SB = DH == 64 ? 2 : 1;
  static constexpr int COL_P = SB * BN, COL_O = COL_P + 2 * (BN / 2);
  static_assert(COL_O + 2 * DH <= TMEM_COLS, "tensor memory");
  static constexpr float RESCALE_GAP = DH == 64 ? 8.f : 0.f;   // log2 of the growth that a reference may lag behind
};

struct Params {
  int B, S, H, Hkv;
  int ld_o;
  float scale_log2;  // (1/sqrt(dh)) * log2(e)
  int causal;
  __nv_bfloat16* O;
  float* lse;
  int* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int DH>
__global__ void __launch_bounds__(THREADS, 1)
attention_fwd_pp_kernel(const __grid_constant__ CUtensorMap tmap, const Params p) {
  using C = Cfg<DH>;
  constexpr int KS = C::KS, VS = C::VS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + 2 * C::Q_BYTES;
  uint8_t* sV = sK + KS * C::KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + VS * C::KV_BYTES);
  uint64_t* q_full = bars;               // [2]
  uint64_t* k_full = q_full + 2;         // [KS]
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;       // [VS]
  uint64_t* v_empty = v_full + VS;
  uint64_t* s_full = v_empty + VS;       // [2] scores of tile t are in tensor memory
  uint64_t* s_free = s_full + 2;         // [SB] the scores that lay in this accumulator are in registers (4 warp arrivals)
  uint64_t* p_full = s_free + 2;         // [2][2] a half of P of tile t is in tensor memory, O is rescaled (4 warp arrivals)
  uint64_t* pv_done = p_full + 4;        // [2] P V of tile t has completed
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(pv_done + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_pairs = (p.S + 2 * BM - 1) / (2 * BM);
  const int pair = n_pairs - 1 - blockIdx.z;  // slowest grid index: longest tiles first over the whole grid
  const int head = blockIdx.x, b = blockIdx.y;
  const int kvh = head / (p.H / p.Hkv);
  const int q0 = pair * 2 * BM;
  const int row_base = b * p.S;
  const int nkv = (p.S + BN - 1) / BN;
  int nb[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int q0t = q0 + t * BM;
    nb[t] = q0t >= p.S ? 0 : (p.causal ? min(q0t / BN + 1, nkv) : nkv);
  }
  const int n_blocks = max(nb[0], nb[1]);
  const int col_q = head * DH;
  const int col_k = (p.H + kvh) * DH;
  const int col_v = (p.H + p.Hkv + kvh) * DH;

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&s_full[t], 1);
      mbar_init(&s_free[t], 4);
      mbar_init(&p_full[2 * t], 4);
      mbar_init(&p_full[2 * t + 1], 4);
      mbar_init(&pv_done[t], 1);
    }
    for (int s = 0; s < KS; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < VS; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) prefetch_tmap(&tmap);
  if (warp == 1) {
    tmem_alloc(tmem_holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_holder), 0);

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
  if (warp == 0) {
    // ------------------------------------ TMA producer ------------------------------------
    if (lane == 0) {
      for (int t = 0; t < 2; ++t) {
        if (nb[t] > 0) {
          mbar_arrive_expect_tx(&q_full[t], C::Q_BYTES);
#pragma unroll
          for (int c = 0; c < C::NCH; ++c)
            tma_load_2d(sQ + t * C::Q_BYTES + c * (BM * 128), &tmap, &q_full[t], col_q + c * 64, row_base + q0 + t * BM);
        }
      }
      int ks = 0, vs = 0;
      uint32_t kph = 0, vph = 0;
      auto load_k = [&](int j) -> bool {
        if (!mbar_wait(&k_empty[ks], kph ^ 1, p.status, ST_TIMEOUT_EMPTY)) return false;
        mbar_arrive_expect_tx(&k_full[ks], C::KV_BYTES);
#pragma unroll
        for (int c = 0; c < C::NCH; ++c)
          tma_load_2d(sK + ks * C::KV_BYTES + c * (BN * 128), &tmap, &k_full[ks], col_k + c * 64, row_base + j * BN);
        if (++ks == KS) { ks = 0; kph ^= 1; }
        return true;
      };
      auto load_v = [&](int j) -> bool {
        if (!mbar_wait(&v_empty[vs], vph ^ 1, p.status, ST_TIMEOUT_EMPTY)) return false;
        mbar_arrive_expect_tx(&v_full[vs], C::KV_BYTES);
#pragma unroll
        for (int c = 0; c < C::NCH; ++c)
          tma_load_2d(sV + vs * C::KV_BYTES + c * (BN * 128), &tmap, &v_full[vs], col_v + c * 64, row_base + j * BN);
        if (++vs == VS) { vs = 0; vph ^= 1; }
        return true;
      };
      // the consumer frees K of block j + 1 before V of block j (its scores come first), so loads go in that order
      bool ok = n_blocks == 0 || load_k(0);
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (j + 1 < n_blocks) ok = load_k(j + 1);
        ok = ok && load_v(j);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------- MMA issuer -------------------------------------
    // The whole warp walks through the loop, so that descriptors and addresses stay in uniform registers; one lane issues. The
    // order is S0(j) PV0(j-1) S1(j) PV1(j-1) S0(j+1) ..., which is the order in which the tiles, half a block apart, need them.
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(BM, BN, false, false);
    constexpr uint32_t idesc_o = make_idesc_bf16(BM, DH, false, true);
    int ks = 0, vs = 0, n_scores = 0;
    uint32_t kph = 0, vph = 0;
    bool ok = true;
    for (int t = 0; t < 2; ++t) ok = ok && (nb[t] == 0 || mbar_wait_warp(&q_full[t], 0, p.status, ST_TIMEOUT_FULL));
    for (int j = 0; j <= n_blocks && ok; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (ok && j < nb[t]) {                         // S = Q K^T of block j
          if (t == 0 || j >= nb[0]) ok = mbar_wait_warp(&k_full[ks], kph, p.status, ST_TIMEOUT_FULL);
          // the scores before these in the same accumulator are in registers
          if (C::SB == 2) ok = ok && (j == 0 || mbar_wait_warp(&s_free[t], (j - 1) & 1, p.status, ST_TIMEOUT_TMEM_EMPTY));
          else ok = ok && (n_scores == 0 || mbar_wait_warp(&s_free[0], (n_scores - 1) & 1, p.status, ST_TIMEOUT_TMEM_EMPTY));
          if (!ok) break;
          ++n_scores;
          tc_fence_after();
          const uint64_t dq = make_smem_desc(smem_u32(sQ + t * C::Q_BYTES), 16, 1024);
          const uint64_t dk = make_smem_desc(smem_u32(sK + ks * C::KV_BYTES), 16, 1024);
          if (leader) {
#pragma unroll
            for (int k = 0; k < DH / 16; ++k) {
              const uint32_t off = (k >> 2) * (BM * 128) + (k & 3) * 32;
              umma_bf16_ss(tmem_base + (C::SB == 2 ? t * BN : 0), smem_desc_at(dq, off), smem_desc_at(dk, off), idesc_s,
                           k > 0 ? 1u : 0u);
            }
            umma_commit(&s_full[t]);
            if (t == 1 || j >= nb[1]) umma_commit(&k_empty[ks]);
          }
          if (t == 1 || j >= nb[1]) {
            if (++ks == KS) { ks = 0; kph ^= 1; }
          }
        }
        if (ok && j > 0 && j - 1 < nb[t]) {            // O (+)= P V of block j - 1
          const int i = j - 1;
          if (t == 0 || i >= nb[0]) ok = mbar_wait_warp(&v_full[vs], vph, p.status, ST_TIMEOUT_FULL);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            ok = ok && mbar_wait_warp(&p_full[2 * t + h], i & 1, p.status, ST_TIMEOUT_MISC);
            if (!ok) break;
            tc_fence_after();
            const uint64_t dv = make_smem_desc(smem_u32(sV + vs * C::KV_BYTES), BN * 128, 1024);
            if (leader) {
#pragma unroll
              for (int k2 = 0; k2 < HALF / 16; ++k2) {
                const int k = h * (HALF / 16) + k2;
                umma_bf16_ts(tmem_base + C::COL_O + t * DH, tmem_base + C::COL_P + t * (BN / 2) + k * 8,
                             smem_desc_at(dv, k * (16 * 128)), idesc_o, (i > 0 || k > 0) ? 1u : 0u);
              }
            }
          }
          if (!ok) break;
          const bool last = t == 1 || i >= nb[1];
          if (leader) {
            umma_commit(&pv_done[t]);
            if (last) umma_commit(&v_empty[vs]);
          }
          if (last) {
            if (++vs == VS) { vs = 0; vph ^= 1; }
          }
        }
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOFTMAX));
    // ------------------------------------ softmax warps ------------------------------------
    const int t = (warp >> 2) - 1;
    const int q = warp & 3;            // TMEM lane quarter this warp may read
    const int r = q * 32 + lane;       // row inside the tile == TMEM lane
    const int q_idx = q0 + t * BM + r; // position inside the sequence
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tm_S = tmem_base + (C::SB == 2 ? t * BN : 0) + lane_off;
    const uint32_t tm_P = tmem_base + C::COL_P + t * (BN / 2) + lane_off;
    const uint32_t tm_O = tmem_base + C::COL_O + t * DH + lane_off;
    const float sl2 = p.scale_log2;
    constexpr float NEG = -1.0e30f;
    float m_ref = NEG, l = 0.f;
    const int n_t = nb[t];
    for (int j = 0; j < n_t; ++j) {
      // Waits in this loop may give up (the status word says so) but do not end it: lanes that left it one by one would be
      // missing at the warp barriers below. Leaving as a whole takes a vote for each wait: 5000 tokens of 32 heads 208 us, 214 with it.
      mbar_wait_converged(&s_full[t], j & 1, p.status, ST_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      uint32_t v[BN];
      __syncwarp();
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32_converged(tm_S + c * 32, v + c * 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[C::SB == 2 ? t : 0]);
      const int kv0 = j * BN;
      const bool need_mask = (p.causal && j == n_t - 1) || (kv0 + BN > p.S);
      const int lim = (p.causal ? min(q_idx, p.S - 1) : (p.S - 1)) - kv0;   // last visible column
      float m4[4] = {NEG, NEG, NEG, NEG};
      if (need_mask) {
        // Masked here and not among the exponentials, where every block would pay a compare and a select per score; the scale
        // is positive (sb_attention_fwd_pp).
#pragma unroll
        for (int i = 0; i < BN; ++i)
          if (i > lim) v[i] = 0xff800000u;             // -inf: 2^x is 0 whatever the row's reference
      }
      {
#pragma unroll
        for (int i = 0; i < BN; i += 2)
          m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      }
      const float m_blk = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl2;
      const bool grow = m_blk > m_ref + C::RESCALE_GAP;   // always true in the first block
      const float alpha = grow ? ex2(m_ref - m_blk) : 1.f;
      if (grow) m_ref = m_blk;
      const float neg_m = -m_ref;
      if (j > 0) {
        // P V of the previous block has read P and updated O
        mbar_wait_converged(&pv_done[t], (j - 1) & 1, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
          for (int c = 0; c < DH / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32_converged(tm_O + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 2) mul2(o[i], o[i + 1], alpha, alpha);
            tmem_st_32x32_converged(tm_O + c * 32, o);
          }
        }
      }
      float sum4[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // exponentials of half a row and their bf16 pairs
        uint32_t pk[HALF / 2];
#pragma unroll
        for (int i2 = 0; i2 < HALF; i2 += 2) {
          const int i = h * HALF + i2;
          fma2(v[i], v[i + 1], sl2, neg_m);
          const float e0 = ex2(__uint_as_float(v[i]));
          const float e1 = ex2(__uint_as_float(v[i + 1]));
          add2(sum4[i & 6], sum4[(i & 6) + 1], __float_as_uint(e0), __float_as_uint(e1));
          pk[i2 >> 1] = pack_bf16x2(e0, e1);
        }
        tmem_st_32x32(tm_P + h * (HALF / 2), pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[2 * t + h]);
      }
      // Roundings are spelt out here and in the log-sum-exp: left to the compiler, what it contracts changes with the code around it.
      const float row_sum = ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3])) + ((sum4[4] + sum4[5]) + (sum4[6] + sum4[7]));
      l = __fadd_rn(__fmul_rn(l, alpha), row_sum);
    }
    if (n_t > 0 && mbar_wait_warp(&pv_done[t], (n_t - 1) & 1, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
#pragma unroll
      for (int c0 = 0; c0 < DH; c0 += 64) {
        uint32_t o[64];
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld_32x32(tm_O + c0 + c * 32, o + c * 32);
        tmem_ld_wait();
        if (q_idx < p.S) {
          const float inv_l = 1.f / l;
          __nv_bfloat16* orow = p.O + static_cast<size_t>(row_base + q_idx) * p.ld_o + head * DH + c0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[c * 8 + 0]) * inv_l, __uint_as_float(o[c * 8 + 1]) * inv_l);
            w.y = pack_bf16x2(__uint_as_float(o[c * 8 + 2]) * inv_l, __uint_as_float(o[c * 8 + 3]) * inv_l);
            w.z = pack_bf16x2(__uint_as_float(o[c * 8 + 4]) * inv_l, __uint_as_float(o[c * 8 + 5]) * inv_l);
            w.w = pack_bf16x2(__uint_as_float(o[c * 8 + 6]) * inv_l, __uint_as_float(o[c * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 8) = w;
          }
        }
        // rows past the end have skipped the stores; the next tensor-memory load needs the whole warp
        if (c0 + 64 < DH) __syncwarp();
      }
      if (q_idx < p.S) {
        if (p.lse)
          p.lse[(static_cast<size_t>(b) * p.H + head) * p.S + q_idx] = __fmaf_rn(m_ref, 0.6931471805599453f, logf(l));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

template <int DH>
static int launch(const CUtensorMap& tm, const Params& p, cudaStream_t stream) {
  auto kern = attention_fwd_pp_kernel<DH>;
  static PerDeviceOnce attr;
  if (allow_smem(attr, kern, Cfg<DH>::SMEM_BYTES, SB_ERR_LAUNCH)) return SB_ERR_LAUNCH;
  dim3 grid(p.H, p.B, (p.S + 2 * BM - 1) / (2 * BM));
  kern<<<grid, THREADS, Cfg<DH>::SMEM_BYTES, stream>>>(tm, p);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

}  // namespace attpp
}  // namespace sb

using namespace sb;

// Same arguments as sb_attention_fwd. The kernel masks scores with -inf, which only a positive scale leaves there (times zero it
// is NaN, times a negative one +inf); a mask behind the scaling costs every call 2 % (5000 tokens of 32 heads 239 -> 245 us
// with a masked and an unmasked loop of exponentials, 250 with one loop in two parts). So other scales go to the one-tile kernel.
extern "C" int sb_attention_fwd_pp(const void* qkv, void* O, float* lse, int B, int S, int H, int Hkv, int dh, int ld,
                                   int ld_o, float scale, int causal, int* status, void* stream_) {
  if (!(scale > 0.f))
    return sb_attention_fwd(qkv, O, lse, B, S, H, Hkv, dh, ld, ld_o, scale, causal, status, stream_);
  if (B <= 0 || S <= 0 || H <= 0 || Hkv <= 0 || (H % Hkv) || (dh != 64 && dh != 128)) return SB_ERR_ARG;
  if (B > 65535 || (S + 127) / 128 > 65535) return SB_ERR_TOO_LARGE;   // grid y / z limits
  if ((ld_o & 7) || (reinterpret_cast<uintptr_t>(O) & 15)) return SB_ERR_ALIGN;
  CUtensorMap tm;
  int rc = make_tmap_2d_bf16(&tm, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(B) * S, ld, 64, 128);
  if (rc) return rc;
  attpp::Params p;
  p.B = B; p.S = S; p.H = H; p.Hkv = Hkv;
  p.ld_o = ld_o;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.O = static_cast<__nv_bfloat16*>(O);
  p.lse = lse;
  p.status = status;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  return dh == 64 ? attpp::launch<64>(tm, p, stream) : attpp::launch<128>(tm, p, stream);
}
