// bf16 GEMM for sm_100a: TMA -> shared memory -> tcgen05.mma -> TMEM -> epilogue.
//
//   C[M,N] = op(A) * op(B)   with fp32 accumulation in tensor memory.
//
// Replaces the three cuBLASLt forms the reference drives (A*B, A*B^T, A^T*B:
// scirust-cuda/src/chain.rs:1037-1083, 1177-1215, 1228-1266) and folds the
// reference's separate residual `add_kernel` (chain.rs:40) into the epilogue.
//
// Operand forms are expressed by the *major-ness* of each operand in memory:
//   A "K-major":  A stored [M, K] row-major (K contiguous)
//   A "MN-major": A stored [K, M] row-major (M contiguous)      (i.e. A^T * ...)
//   B "K-major":  B stored [N, K] row-major (K contiguous)      (i.e. ... * B^T)
//   B "MN-major": B stored [K, N] row-major (N contiguous)
// so  X*W      (W [in,out])  = A K-major,  B MN-major
//     dY*W^T                 = A K-major,  B K-major
//     X^T*dY   (weight grad) = A MN-major, B MN-major
//
// Kernel shape: persistent, one CTA per SM, 10 warps:
//   warp 0   TMA producer (one elected lane)
//   warp 1   MMA issuer (one elected lane); owns the TMEM allocation
//   warp 2-9 epilogue: a warp may touch the 32 TMEM lanes of quarter (warp_id % 4); the two
//            warps of a quarter split the tile's columns
// Two fp32 accumulators (2 x BN columns of TMEM) let the epilogue of tile i overlap the
// main loop of tile i+1. K is walked in a fixed order, so results are bitwise
// repeatable; split-K writes fp32 partials that a second kernel adds in split order.
#include <stdio.h>
#include <algorithm>
#include "sm100_ptx.cuh"
#include "api.h"
#include "per_device.h"
#include "gemm_sched.cuh"

namespace sb {

constexpr int BM = 128;
constexpr int BK = 64;       // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int GEMM_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue

template <int BN>
struct GemmCfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int TMEM_COLS = 2 * BN;  // 512 or 256: both powers of two
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align slack*/ + 256 /*barriers*/;
};

// Convolution operands without a patch matrix. The patches of an NHWC tensor [B, H, W, C] are 4-D TMA boxes of 64 channels
// x a row tile of output pixels, shifted by the filter tap; pixels outside the image arrive as zeros, a stride is the
// map's element stride. Needs C % 64 == 0 and output rows that tile 128 (64 for the weight gradient) pixels. Bound by the
// operand tiles that come out of L2 (each pixel nine times); the patch matrix would cross memory five times per
// convolution. 128 x 32 x 32 x 64 -> 64, 3 x 3: gather + GEMM 133 -> 32 us forward, 61 -> 40 us weight gradient, GEMM +
// scatter 129 -> 33 us input gradient, whose tap sums now stay in fp32.
//   CONV_FPROP  A = patches of x [pixels, taps * C],  B = packed weights [oc, taps * C]
//   CONV_WGRAD  A = dy [pixels, oc] (transposed),     B = patches of x
//   CONV_DGRAD  A = patches of dy, taps mirrored (stride 1), B = packed weights read as [oc, C] per tap
enum { CONV_NONE = 0, CONV_FPROP = 1, CONV_WGRAD = 2, CONV_DGRAD = 3 };
struct ConvTile {
  int cb;              // 64-channel blocks per tap of the tensor that is patched
  int C;               // channels of x (DGRAD: columns of one tap in the packed weights)
  int KW, stride, pad; // filter width (a square filter), stride and padding of the convolution
  int ow, ohw;         // output pixels per row and per image of the pixel grid that is walked
};

struct GemmParams {
  int M, N, K;
  int splits;          // explicit split-K factor (1 = none)
  int kb_per_split;    // k-blocks per split
  void* C;             // bf16 [M, ldc] when splits == 1; fp32 [splits, M, N] partials otherwise
  int ldc;
  const void* R;       // optional bf16 residual [M, ldr] added in the epilogue (splits == 1)
  int ldr;
  int* status;
  BalancedSched sched;   // balanced schedule (splits == 1 only); see gemm_sched.cuh
  float* partials;       // scratch slots of the balanced schedule: dense fp32 [BM, BN] blocks
  ConvTile conv;
};

// Patch box of output pixels [pix, pix + box) at k-block / column block `blk` (tap-major, 64 channels each).
template <int CONV>
__device__ __forceinline__ void conv_load_patch(void* dst, const CUtensorMap* m, uint64_t* bar, const ConvTile& cv,
                                                int pix, int blk) {
  const int tap = blk / cv.cb, c0 = (blk - tap * cv.cb) * 64;
  const int kh = tap / cv.KW, kw = tap - kh * cv.KW;
  const int b0 = pix / cv.ohw, oh0 = (pix - b0 * cv.ohw) / cv.ow;
  if constexpr (CONV == CONV_DGRAD) tma_load_4d(dst, m, bar, c0, cv.pad - kw, oh0 + cv.pad - kh, b0);
  else tma_load_4d(dst, m, bar, c0, kw - cv.pad, oh0 * cv.stride + kh - cv.pad, b0);
}

template <int BN, bool A_MN, bool B_MN, int CONV = CONV_NONE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const GemmParams p) {
  using Cfg = GemmCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  // 128B-swizzled tiles need 1024-byte alignment.
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* tmem_full = empty_bar + Cfg::STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;

  const int mt = (p.M + BM - 1) / BM;
  const int nt = (p.N + BN - 1) / BN;
  const int num_kb = (p.K + BK - 1) / BK;
  const int tiles_mn = mt * nt;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8);  // one arrival per epilogue warp
    }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_holder), 0);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      SegIter iter(p.sched, blockIdx.x, gridDim.x, tiles_mn, num_kb, p.splits, p.kb_per_split);
      Seg sg;
      while (ok && iter.next(sg)) {
        const int n_idx = sg.tile / mt;
        const int m_idx = sg.tile - n_idx * mt;
        const int kb0 = sg.kb0, kb1 = sg.kb1;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* sa = tiles + stage * Cfg::STAGE_BYTES;
          uint8_t* sb_ = sa + Cfg::A_BYTES;
          mbar_arrive_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES);
          if constexpr (CONV == CONV_FPROP || CONV == CONV_DGRAD) {
            conv_load_patch<CONV>(sa, &tmap_a, &full_bar[stage], p.conv, m_idx * BM, kb);
          } else if constexpr (!A_MN) {
            tma_load_2d(sa, &tmap_a, &full_bar[stage], kb * BK, m_idx * BM);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c)
              tma_load_2d(sa + c * (64 * BK * 2), &tmap_a, &full_bar[stage], m_idx * BM + c * 64, kb * BK);
          }
          if constexpr (CONV == CONV_WGRAD) {
            const int last = p.N / 64 - 1;            // columns past N are dropped by the epilogue: any block will do
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              conv_load_patch<CONV>(sb_ + c * (64 * BK * 2), &tmap_b, &full_bar[stage], p.conv, kb * BK,
                                    min(n_idx * (BN / 64) + c, last));
          } else if constexpr (CONV == CONV_DGRAD) {
            const int tap = kb / p.conv.cb;
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              tma_load_2d(sb_ + c * (64 * BK * 2), &tmap_b, &full_bar[stage], tap * p.conv.C + n_idx * BN + c * 64,
                          (kb - tap * p.conv.cb) * 64);
          } else if constexpr (!B_MN) {
            tma_load_2d(sb_, &tmap_b, &full_bar[stage], kb * BK, n_idx * BN);
          } else {
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              tma_load_2d(sb_ + c * (64 * BK * 2), &tmap_b, &full_bar[stage], n_idx * BN + c * 64, kb * BK);
          }
          if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    {
      // The whole warp walks through the loop and one lane issues: descriptors and addresses then stay in uniform registers.
      // As the loop of a single thread a product took 70 to 150 cycles to issue, as long as a narrow one runs.
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int it = 0;
      SegIter iter(p.sched, blockIdx.x, gridDim.x, tiles_mn, num_kb, p.splits, p.kb_per_split);
      Seg sg;
      for (; ok && iter.next(sg); ++it) {
        const int kb0 = sg.kb0, kb1 = sg.kb1;
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_warp(&tmem_empty[acc], acc_phase ^ 1, p.status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * Cfg::STAGE_BYTES);
          const uint64_t da = make_smem_desc(sa, A_MN ? 64 * BK * 2 : 16, 1024);
          const uint64_t db = make_smem_desc(sa + Cfg::A_BYTES, B_MN ? 64 * BK * 2 : 16, 1024);
          if (leader) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16_ss(d_tmem, smem_desc_at(da, k * (A_MN ? UMMA_K * 128 : UMMA_K * 2)),
                           smem_desc_at(db, k * (B_MN ? UMMA_K * 128 : UMMA_K * 2)), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            umma_commit(&empty_bar[stage]);  // frees the stage once these MMAs have read it
          }
          if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && leader) umma_commit(&tmem_full[acc]);
        __syncwarp();
      }
    }
  } else {
    // -------------------------------- epilogue --------------------------------
    const int q = warp & 3;            // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;  // which half of the tile's columns this warp drains
    bool ok = true;
    int it = 0;
    SegIter iter(p.sched, blockIdx.x, gridDim.x, tiles_mn, num_kb, p.splits, p.kb_per_split);
    Seg sg;
    for (; ok && iter.next(sg); ++it) {
      const int split = sg.split;
      const int n_idx = sg.tile / mt;
      const int m_idx = sg.tile - n_idx * mt;
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait_warp(&tmem_full[acc], acc_phase, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int row = m_idx * BM + q * 32 + lane;
      const uint32_t taddr_row = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr_row + c * 32, r);
        tmem_ld_wait();
        const int col0 = n_idx * BN + c * 32;
        if (sg.slot >= 0) {
          // part of a tile of the balanced schedule: dense fp32 block, finished by the fix-up kernel
          float* prow = p.partials + (static_cast<size_t>(sg.slot) * BM + (q * 32 + lane)) * BN + c * 32;
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<uint4*>(prow + v * 4) = make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
        } else if (row < p.M && col0 < p.N) {
          if (p.splits == 1) {
            __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<size_t>(row) * p.ldc + col0;
            const __nv_bfloat16* rrow =
                p.R ? reinterpret_cast<const __nv_bfloat16*>(p.R) + static_cast<size_t>(row) * p.ldr + col0
                    : nullptr;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              if (col0 + v * 8 < p.N) {  // N % 8 == 0 is enforced on the host
                float f[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
                if (rrow) {
                  const uint4 rv = *reinterpret_cast<const uint4*>(rrow + v * 8);
                  f[0] += bf16_lo(rv.x); f[1] += bf16_hi(rv.x);
                  f[2] += bf16_lo(rv.y); f[3] += bf16_hi(rv.y);
                  f[4] += bf16_lo(rv.z); f[5] += bf16_hi(rv.z);
                  f[6] += bf16_lo(rv.w); f[7] += bf16_hi(rv.w);
                }
                uint4 o;
                o.x = pack_bf16x2(f[0], f[1]);
                o.y = pack_bf16x2(f[2], f[3]);
                o.z = pack_bf16x2(f[4], f[5]);
                o.w = pack_bf16x2(f[6], f[7]);
                *reinterpret_cast<uint4*>(crow + v * 8) = o;
              }
            }
          } else {
            float* prow = reinterpret_cast<float*>(p.C) +
                          (static_cast<size_t>(split) * p.M + row) * static_cast<size_t>(p.N) + col0;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              if (col0 + v * 4 < p.N) {  // N % 8 == 0
                *reinterpret_cast<uint4*>(prow + v * 4) =
                    make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
    }
  }

  // Teardown: every role loop above is bounded, so all threads arrive here.
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

// Adds split-K partials in split order 0..S-1 (fixed order => bitwise repeatable),
// optionally adds a bf16 residual, rounds to bf16 (F32: leaves the sums as they are). U partials are on their way at once: eight
// from four splits on (a weight gradient of a convolution has up to 64 and few elements: 49 splits of 64 x 576 8.3 us with one at a
// time, 6.1 with eight), one for fewer, where the unused places of eight cost (product and sum, us, one / eight: two splits, 999 x 1536 x
// 1024 18.0 / 19.0; three, 300 x 4096 x 4096 19.25 / 19.35).
template <bool F32, int U>
__global__ void splitk_reduce_kernel(const float* __restrict__ part, int splits, size_t mn, int N, void* __restrict__ C_, int ldc,
                                     const __nv_bfloat16* __restrict__ R, int ldr) {
  const size_t i4 = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (i4 >= mn) return;
  float4 acc = __ldg(reinterpret_cast<const float4*>(part + i4));
  for (int s0 = 1; s0 < splits; s0 += U) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s0 + u < splits) v[u] = __ldg(reinterpret_cast<const float4*>(part + (s0 + u) * mn + i4));
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s0 + u < splits) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
  }
  const size_t row = i4 / N;
  const int col = static_cast<int>(i4 - row * N);
  if (R) {
    const uint2 rv = *reinterpret_cast<const uint2*>(R + row * ldr + col);
    acc.x += bf16_lo(rv.x); acc.y += bf16_hi(rv.x);
    acc.z += bf16_lo(rv.y); acc.w += bf16_hi(rv.y);
  }
  if (F32) {
    *reinterpret_cast<float4*>(static_cast<float*>(C_) + row * ldc + col) = acc;
  } else {
    uint2 o;
    o.x = pack_bf16x2(acc.x, acc.y);
    o.y = pack_bf16x2(acc.z, acc.w);
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(C_) + row * ldc + col) = o;
  }
}

template <bool F32>
static auto splitk_reduce(int splits) { return splits < 4 ? splitk_reduce_kernel<F32, 1> : splitk_reduce_kernel<F32, 8>; }

// ------------------------------ host side ------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  // cuTensorMapEncodeTiled is a driver call and wants a context current on the calling thread. A thread that has
  // only ever used device 0 through a framework that skips cudaSetDevice when "the device is already 0" (an autograd
  // worker whose first native call is a tensor-map encode) has none: bind the primary context once per thread.
  thread_local bool context_bound = false;
  if (!context_bound) {
    cudaFree(nullptr);
    context_bound = true;
  }
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
      fprintf(stderr, "scirust_b200: cuTensorMapEncodeTiled could not be resolved\n");
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// 2-D bf16 tensor map with 128B swizzle. `inner` elements are contiguous; `ld` is
// the row pitch in elements. Returns 0 on success.
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return SB_ERR_DRIVER;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || ((ld * 2) & 15)) return SB_ERR_ALIGN;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    fprintf(stderr, "scirust_b200: tensor map refused (driver code %d): base %p, dims %llu x %llu, pitch %llu B, box %u x %u\n",
            static_cast<int>(r), base, static_cast<unsigned long long>(inner), static_cast<unsigned long long>(outer),
            static_cast<unsigned long long>(ld * 2), box_inner, box_outer);
  return r == CUDA_SUCCESS ? 0 : SB_ERR_DRIVER;
}

// 3-D bf16 tensor map with 128B swizzle: dims (d0 contiguous, d1, d2), pitches in elements; the box is
// box0 x box1 x 1. Out-of-range parts of a box are zero on loads and dropped on stores.
int make_tmap_3d_bf16(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t pitch1,
                      uint64_t pitch2, uint32_t box0, uint32_t box1) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return SB_ERR_DRIVER;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || ((pitch1 * 2) & 15) || ((pitch2 * 2) & 15)) return SB_ERR_ALIGN;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {pitch1 * 2, pitch2 * 2};
  cuuint32_t box[3] = {box0, box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : SB_ERR_DRIVER;
}

// 2-D tensor map over 16-bit words without swizzle (row-major copy of a box into shared memory).
// Used by the weight-streaming kernels: `inner` 2-byte words are contiguous, `pitch_bytes` is the row
// pitch. Out-of-range parts of a box are filled with zeros.
int make_tmap_2d_u16_plain(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t pitch_bytes,
                           uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return SB_ERR_DRIVER;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (pitch_bytes & 15)) return SB_ERR_ALIGN;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {pitch_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : SB_ERR_DRIVER;
}

// Patches of an NHWC tensor [B, H, W, C]: boxes of 64 channels x `box` output pixels (ow per row, whole rows, whole
// images when an image is smaller than the box) at element stride `stride`. 0 when the shape does not tile.
static int make_tmap_patches(CUtensorMap* out, const void* base, int B, int H, int W, int C, int ow, int oh, int stride,
                             int box) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return SB_ERR_DRIVER;
  if (reinterpret_cast<uintptr_t>(base) & 15) return SB_ERR_ALIGN;
  if (ow > box || box % ow || (C & 63)) return SB_ERR_ARG;
  int rows = box / ow, images = 1;
  if (rows > oh) {
    if (rows % oh) return SB_ERR_ARG;
    images = rows / oh;
    rows = oh;
  } else if (oh % rows) {
    return SB_ERR_ARG;
  }
  const cuuint64_t c = static_cast<cuuint64_t>(C);
  cuuint64_t dims[4] = {c, static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(H), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {c * 2, c * 2 * W, c * 2 * W * H};
  cuuint32_t bx[4] = {64, static_cast<cuuint32_t>((ow - 1) * stride + 1), static_cast<cuuint32_t>((rows - 1) * stride + 1),
                      static_cast<cuuint32_t>(images)};
  cuuint32_t es[4] = {1, static_cast<cuuint32_t>(stride), static_cast<cuuint32_t>(stride), 1};
  if (bx[1] > 256 || bx[2] > 256 || stride > 8) return SB_ERR_ARG;
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, bx, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : SB_ERR_DRIVER;
}

static int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_num_sms;
}

template <int BN, bool A_MN, bool B_MN, int CONV = CONV_NONE>
static int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                       cudaStream_t stream) {
  using Cfg = GemmCfg<BN>;
  auto kern = gemm_bf16_kernel<BN, A_MN, B_MN, CONV>;
  static PerDeviceOnce attr;
  if (allow_smem(attr, kern, Cfg::SMEM_BYTES, SB_ERR_LAUNCH)) return SB_ERR_LAUNCH;
  kern<<<grid, GEMM_THREADS, Cfg::SMEM_BYTES, stream>>>(ta, tb, p);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

}  // namespace sb

using namespace sb;

// C[M,N] (bf16, pitch ldc) = op(A) op(B) (+ R).  a_mn / b_mn select the operand
// major-ness described at the top of this file; lda/ldb are row pitches (elements)
// of the matrices as stored. `splits` > 1 is explicit split-K and needs `workspace` of
// splits*M*N floats. `splits` == 0 selects the balanced schedule (whole waves of tiles one per
// CTA, the k-blocks of the last partial wave dealt out evenly over all SMs); it needs `workspace`
// of sb_gemm_balanced_workspace_floats() floats and falls back to one tile per CTA without it.
// bn: 0 = choose, else 128 or 256.
extern "C" size_t sb_gemm_balanced_workspace_floats() { return static_cast<size_t>(num_sms()) * 3 * BM * 256; }

extern "C" int sb_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda,
                            int ldb, int ldc, int ldr, int a_mn, int b_mn, int splits, void* workspace, int bn,
                            int* status, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return SB_ERR_ARG;
  if ((N & 7) || (ldc & 7) || (R && (ldr & 7))) return SB_ERR_ALIGN;
  if (reinterpret_cast<uintptr_t>(C) & 15) return SB_ERR_ALIGN;
  if (R && (reinterpret_cast<uintptr_t>(R) & 15)) return SB_ERR_ALIGN;
  const int num_kb = (K + BK - 1) / BK;
  const bool balanced = splits == 0 && workspace != nullptr;
  if (splits < 1) splits = 1;
  if (splits > num_kb) splits = num_kb;
  int kb_per_split = (num_kb + splits - 1) / splits;
  splits = (num_kb + kb_per_split - 1) / kb_per_split;  // no empty split
  if (splits > 1 && !workspace) return SB_ERR_ARG;
  if (bn == 0) bn = (N <= 128) ? 128 : 256;
  if (bn != 128 && bn != 256) return SB_ERR_ARG;

  CUtensorMap ta, tb;
  int rc;
  if (!a_mn) rc = make_tmap_2d_bf16(&ta, A, K, M, lda, BK, BM);
  else rc = make_tmap_2d_bf16(&ta, A, M, K, lda, 64, BK);
  if (rc) return rc;
  if (!b_mn) rc = make_tmap_2d_bf16(&tb, B, K, N, ldb, BK, bn);
  else rc = make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, BK);
  if (rc) return rc;

  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.splits = splits;
  p.kb_per_split = kb_per_split;
  p.C = splits > 1 ? workspace : C;
  p.ldc = ldc;
  p.R = splits > 1 ? nullptr : R;
  p.ldr = ldr;
  p.status = status;
  p.partials = nullptr;
  const int mt = (M + BM - 1) / BM, nt = (N + bn - 1) / bn;
  const int tiles = mt * nt * splits;
  int grid = tiles < num_sms() ? tiles : num_sms();
  bool fixup = false;
  if (balanced && plan_balanced(tiles, num_kb, num_sms(), &p.sched, &fixup)) {
    p.partials = static_cast<float*>(workspace);
    grid = p.sched.dp_tiles > 0 ? num_sms() : p.sched.sk_workers;
  } else {
    p.sched.dp_tiles = p.sched.sk_tiles = p.sched.sk_workers = p.sched.sk_slots = 0;
  }

#define SB_DISPATCH(BN_)                                                                   \
  do {                                                                                     \
    if (!a_mn && !b_mn) rc = launch_gemm<BN_, false, false>(ta, tb, p, grid, stream);      \
    else if (!a_mn && b_mn) rc = launch_gemm<BN_, false, true>(ta, tb, p, grid, stream);   \
    else if (a_mn && !b_mn) rc = launch_gemm<BN_, true, false>(ta, tb, p, grid, stream);   \
    else rc = launch_gemm<BN_, true, true>(ta, tb, p, grid, stream);                       \
  } while (0)
  if (bn == 256) SB_DISPATCH(256); else SB_DISPATCH(128);
#undef SB_DISPATCH
  if (rc) return rc;

  if (fixup) {
    dim3 fg(p.sched.sk_tiles, BM * bn / (256 * 4));
    __nv_bfloat16* c = static_cast<__nv_bfloat16*>(C);
    const __nv_bfloat16* r = static_cast<const __nv_bfloat16*>(R);
    if (bn == 256) balanced_fixup_kernel<BM, 256><<<fg, 256, 0, stream>>>(p.sched, p.partials, c, ldc, r, ldr, M, N, mt, num_kb);
    else balanced_fixup_kernel<BM, 128><<<fg, 256, 0, stream>>>(p.sched, p.partials, c, ldc, r, ldr, M, N, mt, num_kb);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  }
  if (splits > 1) {
    const size_t mn = static_cast<size_t>(M) * N;
    const int threads = 256;
    const unsigned blocks = static_cast<unsigned>((mn / 4 + threads - 1) / threads);
    auto kern = splitk_reduce<false>(splits);
    kern<<<blocks, threads, 0, stream>>>(static_cast<const float*>(workspace), splits, mn, N, C, ldc,
                                         static_cast<const __nv_bfloat16*>(R), ldr);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  }
  return 0;
}

// A plain copy of 16-byte words, four in flight per thread: as a kernel it costs the host half of what cudaMemcpyAsync does.
__global__ void __launch_bounds__(256) copy_words_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, size_t words) {
  const size_t step = static_cast<size_t>(gridDim.x) * 1024;
  for (size_t i = static_cast<size_t>(blockIdx.x) * 1024 + threadIdx.x; i < words; i += step) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * 256 < words) v[u] = __ldg(src + i + u * 256);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * 256 < words) dst[i + u * 256] = v[u];
  }
}

// One product of an NHWC convolution (square k x k filter) without a patch matrix; the packed weights are [oc, k*k*C] in
// (kh, kw, c) order, C % 64 == 0, oc % 64 == 0.
//   mode 1: out = y [B*OH*OW, oc]   from a = x, b = weights
//   mode 2: out = dw [oc, k*k*C]    from a = dy [B*OH*OW, oc], b = x
//   mode 3: out = dx [B*H*W, C]     from a = dy, b = weights; stride 1
//   mode 4: mode 2 with an fp32 out; splits > 1 only (SB_ERR_ARG without), where the sum of the splits is fp32 anyway
// splits > 1: split-K over `workspace` (splits * rows * columns of out, floats). Shapes whose pixel rows do not tile 128
// (mode 2: 64) pixels are refused with SB_ERR_ARG. keep (mode 1, optional): gets a copy of x.
static int conv_gemm(int mode, const void* a, const void* b, void* out, void* keep, int B, int H, int W, int C, int oc, int k,
                     int stride, int pad, int OH, int OW, int splits, void* workspace, int* status, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const bool f32 = mode == 4;
  if (f32) mode = 2;
  if (mode < 1 || mode > 3 || B <= 0 || C <= 0 || oc <= 0 || (C & 63) || (oc & 63) || k < 1 || stride < 1 || pad < 0 || !status)
    return SB_ERR_ARG;
  if (OH != (H + 2 * pad - k) / stride + 1 || OW != (W + 2 * pad - k) / stride + 1 || OH < 1 || OW < 1) return SB_ERR_ARG;
  if (mode == 3 && stride != 1) return SB_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(keep)) & 15) return SB_ERR_ALIGN;
  const int taps = k * k, kp = taps * C;
  const long long pix_o = static_cast<long long>(B) * OH * OW, pix_i = static_cast<long long>(B) * H * W;
  if (pix_o >= (1ll << 31) || pix_i >= (1ll << 31)) return SB_ERR_TOO_LARGE;
  GemmParams p;
  p.M = mode == 2 ? oc : static_cast<int>(mode == 1 ? pix_o : pix_i);
  p.N = mode == 1 ? oc : mode == 2 ? kp : C;
  p.K = mode == 1 ? kp : mode == 2 ? static_cast<int>(pix_o) : taps * oc;
  const int num_kb = (p.K + BK - 1) / BK;
  if (splits < 1) splits = 1;
  if (splits > num_kb) splits = num_kb;
  p.kb_per_split = (num_kb + splits - 1) / splits;
  splits = (num_kb + p.kb_per_split - 1) / p.kb_per_split;
  if ((splits > 1 && !workspace) || (f32 && splits == 1)) return SB_ERR_ARG;
  const int bn = p.N <= 128 ? 128 : 256;
  p.splits = splits;
  p.C = splits > 1 ? workspace : out;
  p.ldc = p.N;
  p.R = nullptr; p.ldr = 0;
  p.status = status;
  p.partials = nullptr;
  p.sched.dp_tiles = p.sched.sk_tiles = p.sched.sk_workers = p.sched.sk_slots = 0;
  p.conv.C = C; p.conv.KW = k; p.conv.stride = stride; p.conv.pad = pad;
  p.conv.cb = (mode == 3 ? oc : C) / 64;
  p.conv.ow = mode == 3 ? W : OW;
  p.conv.ohw = mode == 3 ? H * W : OH * OW;
  CUtensorMap ta, tb;
  int rc;
  if (mode == 1) {
    rc = make_tmap_patches(&ta, a, B, H, W, C, OW, OH, stride, BM);
    if (!rc) rc = make_tmap_2d_bf16(&tb, b, kp, oc, kp, BK, bn);
  } else if (mode == 2) {
    rc = make_tmap_2d_bf16(&ta, a, oc, pix_o, oc, 64, BK);
    if (!rc) rc = make_tmap_patches(&tb, b, B, H, W, C, OW, OH, stride, BK);
  } else {
    rc = make_tmap_patches(&ta, a, B, OH, OW, oc, W, H, 1, BM);
    if (!rc) rc = make_tmap_2d_bf16(&tb, b, kp, oc, kp, 64, BK);
  }
  if (rc) return rc;
  if (keep) {
    const size_t words = static_cast<size_t>(pix_i) * C / 8;
    copy_words_kernel<<<static_cast<unsigned>(std::min<size_t>((words + 1023) / 1024, 8 * num_sms())), 256, 0, stream>>>(
        static_cast<const uint4*>(a), static_cast<uint4*>(keep), words);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  }
  const long long tiles = static_cast<long long>((p.M + BM - 1) / BM) * ((p.N + bn - 1) / bn) * splits;
  const int grid = tiles < num_sms() ? static_cast<int>(tiles) : num_sms();
  if (mode == 1) rc = bn == 128 ? launch_gemm<128, false, false, CONV_FPROP>(ta, tb, p, grid, stream)
                                : launch_gemm<256, false, false, CONV_FPROP>(ta, tb, p, grid, stream);
  else if (mode == 2) rc = bn == 128 ? launch_gemm<128, true, true, CONV_WGRAD>(ta, tb, p, grid, stream)
                                     : launch_gemm<256, true, true, CONV_WGRAD>(ta, tb, p, grid, stream);
  else rc = bn == 128 ? launch_gemm<128, false, true, CONV_DGRAD>(ta, tb, p, grid, stream)
                      : launch_gemm<256, false, true, CONV_DGRAD>(ta, tb, p, grid, stream);
  if (rc) return rc;
  if (splits > 1) {
    const size_t mn = static_cast<size_t>(p.M) * p.N;
    auto kern = f32 ? splitk_reduce<true>(splits) : splitk_reduce<false>(splits);
    kern<<<static_cast<unsigned>((mn / 4 + 255) / 256), 256, 0, stream>>>(static_cast<const float*>(workspace), splits, mn, p.N, out,
                                                                          p.N, nullptr, 0);
    if (cudaGetLastError() != cudaSuccess) return SB_ERR_LAUNCH;
  }
  return 0;
}

extern "C" int sb_conv_gemm(int mode, const void* a, const void* b, void* out, int B, int H, int W, int C, int oc, int k,
                            int stride, int pad, int OH, int OW, int splits, void* workspace, int* status,
                            void* stream_) {
  return conv_gemm(mode, a, b, out, nullptr, B, H, W, C, oc, k, stride, pad, OH, OW, splits, workspace, status, stream_);
}

// Mode 1 with a copy of x into keep [B*H*W, C], for a weight gradient that is taken later.
extern "C" int sb_conv_fprop_keep(const void* x, const void* w, void* y, void* keep, int B, int H, int W, int C, int oc, int k,
                                  int stride, int pad, int OH, int OW, int splits, void* workspace, int* status,
                                  void* stream_) {
  if (!keep) return SB_ERR_ARG;
  return conv_gemm(1, x, w, y, keep, B, H, W, C, oc, k, stride, pad, OH, OW, splits, workspace, status, stream_);
}
