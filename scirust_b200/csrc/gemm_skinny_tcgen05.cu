// Weight-streaming GEMM for batched decoding: C[rows, N] = X[rows, K] . W (+ R) with 9..64 activation rows.
//
// With so few rows the product is bound by the weight bytes, and on this GPU a copy only reaches the HBM rate with
// about 30 MB in flight (the loaded latency is several microseconds). The general GEMM spends its shared memory on
// 128-row activation tiles that are mostly zero fill and keeps 128 KB of weights in flight per SM; here the roles are
// swapped: the WEIGHT tile is the 128-row MMA operand (128 output columns x one k-block, 16 KB), the activations
// are the narrow operand (16 / 32 / 64 rows x one k-block, 2-8 KB), so 9 to 12 stages fit (144-192 KB of weights in
// flight per SM) and every weight byte is read exactly once. The accumulator is C^T (lane = output column, TMEM
// column = activation row); the epilogue writes it back transposed.
//
//   bf16 (I8 = false): W [K, N] as stored (N contiguous) is the MN-major A operand, X [rows, K] the K-major B
//                      operand; tcgen05.mma.kind::f16, fp32 accumulation, k walked in ascending order.
//   int8 (I8 = true):  W8A8 of the reference's quantised linear layer (scirust-core/src/quantization.rs:150-190):
//                      weights as the transposed codes [N, K], activations quantised per row; kind::i8, int32
//                      accumulation (exact), one rescale by sx[m] * sw[n].
// Split-K partials (fp32 / int32) are added in split order: inside a thread-block cluster, whose CTAs are the splits of one
// column tile, where all these clusters are on the GPU at once (it holds 33 of four CTAs, 45 of three), else by
// skinny_reduce_kernel from [split][row][N] in memory. Us with that kernel / in the cluster, in a chain of dependent launches:
// 4096 x 4096, 16 rows 8.6 / 8.2, 64 rows 11.1 / 9.2, int8 11.9 / 9.9; 14336 x 4096, 64 rows 24.5 / 22.0, int8 17.2 / 15.7; 1024 x
// 1024, 64 int8 rows 8.0 / 7.4. The 48 tiles of a 6144-wide product in three splits are three too many for it.
// Warps: 0 TMA, 1 MMA, 2-5 epilogue (one per TMEM lane quarter).
#include "sm100_ptx.cuh"
#include "api.h"
#include "per_device.h"
#include "dependent.cuh"
#include <atomic>

namespace sb {

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);
int num_sms();

constexpr int SK_BM = 128;          // output columns per tile (the MMA's M)
constexpr int SK_THREADS = 192;
constexpr int SK_MAX_CLUSTER = 6;   // splits that finish in a cluster
constexpr int SK_A_BYTES = 16384;   // 128 columns x (64 bf16 | 128 int8) of k

template <int RB>
struct SkinnyCfg {
  static constexpr int B_BYTES = RB * 128;
  static constexpr int STAGE_BYTES = SK_A_BYTES + B_BYTES;
  static constexpr int STAGES = (227 * 1024 - 1280) / STAGE_BYTES;
  static constexpr int ACC_STRIDE = RB < 32 ? 32 : RB;       // TMEM columns between the two accumulators
  static constexpr int TMEM_COLS = 2 * ACC_STRIDE;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

struct SkinnyParams {
  int rows, N, K;
  int splits, kb_per_split;
  void* C; int ldc;               // bf16 [rows, ldc]; or partials [splits][rows][N] (fp32 / int32)
  const void* R; int ldr;
  const float* sx; const float* sw;   // int8 only
  int* status;
};

__host__ __device__ constexpr uint32_t skinny_idesc(bool i8, int n) {
  // kind::f16: D f32 (1 << 4), A / B bf16 (1 << 7, 1 << 10), A MN-major (1 << 15);  kind::i8: D s32 (2 << 4), A / B s8
  return (i8 ? ((2u << 4) | (1u << 7) | (1u << 10)) : ((1u << 4) | (1u << 7) | (1u << 10) | (1u << 15))) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(SK_BM >> 4) << 24);
}

template <bool I8>
__device__ __forceinline__ void skinny_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  if constexpr (I8) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  }
}

template <int RB, bool I8, bool CLUSTER>
__global__ void __launch_bounds__(SK_THREADS, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const SkinnyParams p) {
  using Cfg = SkinnyCfg<RB>;
  constexpr int BKE = I8 ? 128 : 64;                      // k elements per k-block (128 bytes of k for both types)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* tmem_full = empty_bar + Cfg::STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nt = (p.N + SK_BM - 1) / SK_BM;
  const int num_kb = (p.K + BKE - 1) / BKE;
  // CLUSTER: grid (column tiles, splits), one item per CTA; else a CTA walks over items split-major
  const int items = nt * p.splits;
  const int first = CLUSTER ? blockIdx.y * nt + blockIdx.x : blockIdx.x, step = CLUSTER ? items : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], 4); }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 0 && lane == 0) { prefetch_tmap(&tmap_w); prefetch_tmap(&tmap_x); }
  if (warp == 1) { tmem_alloc(tmem_holder, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_holder), 0);
  // Launched while the small kernels ahead of it (norm, quantiser, split sums) still run, a CTA brings as much of its
  // weights into L2 as its ring will hold. More takes the memory from the kernel ahead: a layer of 64 rows at Llama-3-8B
  // shape 218.4 us without, 214.2 with 8 k-blocks, 215.2 with 16, 225.2 with 64; 16 int8 rows 123.2 / 120.0 / 119.2 / 118.3.
  pdl_trigger();
  if (warp == 0 && lane == 0) {
    const int split = first / nt, n_idx = first - split * nt;
    const int kb0 = split * p.kb_per_split, kb1 = min(min(num_kb, kb0 + p.kb_per_split), kb0 + Cfg::STAGES);
    for (int kb = kb0; kb < kb1; ++kb) {
      if constexpr (I8) {
        tma_prefetch_2d(&tmap_w, kb * 64, n_idx * SK_BM);
      } else {
        tma_prefetch_2d(&tmap_w, n_idx * SK_BM, kb * 64);
        tma_prefetch_2d(&tmap_w, n_idx * SK_BM + 64, kb * 64);
      }
    }
  }
  __syncwarp();
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = first; t < items && ok; t += step) {
        const int split = t / nt, n_idx = t - split * nt;
        const int kb0 = split * p.kb_per_split, kb1 = min(num_kb, kb0 + p.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* sa = tiles + stage * Cfg::STAGE_BYTES;
          uint8_t* sb_ = sa + SK_A_BYTES;
          mbar_arrive_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES);
          if constexpr (I8) {
            // both maps are over 16-bit words (two int8 each): x = k / 2, boxes of 64 words = 128 bytes of k
            tma_load_2d(sa, &tmap_w, &full_bar[stage], kb * 64, n_idx * SK_BM);
            tma_load_2d(sb_, &tmap_x, &full_bar[stage], kb * 64, 0);
          } else {
            // W [K, N]: two boxes of 64 k x 64 columns (MN-major operand); X [rows, K]: one box of RB rows x 64 k
            tma_load_2d(sa, &tmap_w, &full_bar[stage], n_idx * SK_BM, kb * 64);
            tma_load_2d(sa + 8192, &tmap_w, &full_bar[stage], n_idx * SK_BM + 64, kb * 64);
            tma_load_2d(sb_, &tmap_x, &full_bar[stage], kb * 64, 0);
          }
          if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    {
      // The whole warp walks through the loop and one lane issues: descriptors and addresses then stay in uniform registers.
      // As the loop of a single thread a product took 70 to 150 cycles to issue, as long as a narrow one runs.
      const bool leader = elect_one();
      constexpr uint32_t idesc = skinny_idesc(I8, RB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int it = 0;
      for (int t = first; t < items && ok; t += step, ++it) {
        const int split = t / nt;
        const int kb0 = split * p.kb_per_split, kb1 = min(num_kb, kb0 + p.kb_per_split);
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_warp(&tmem_empty[acc], acc_phase ^ 1, p.status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * Cfg::ACC_STRIDE;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * Cfg::STAGE_BYTES);
          const uint64_t da = make_smem_desc(sa, I8 ? 16 : 64 * 64 * 2, 1024), db = make_smem_desc(sa + SK_A_BYTES, 16, 1024);
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k)                 // four MMAs of 32 bytes of k each
              skinny_mma<I8>(d_tmem, smem_desc_at(da, k * (I8 ? 32 : 16 * 128)), smem_desc_at(db, k * 32), idesc,
                             (kb > kb0 || k > 0) ? 1u : 0u);
            umma_commit(&empty_bar[stage]);
          }
          if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && leader) umma_commit(&tmem_full[acc]);
        __syncwarp();
      }
    }
  } else {
    const int q = warp & 3;                             // warps 2, 3, 4, 5 -> lane quarters 2, 3, 0, 1
    bool ok = true;
    int it = 0;
    for (int t = first; t < items && ok; t += step, ++it) {
      const int split = t / nt, n_idx = t - split * nt;
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait_warp(&tmem_full[acc], acc_phase, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int col = n_idx * SK_BM + q * 32 + lane;    // this thread's output column
      const uint32_t taddr = tmem_base + acc * Cfg::ACC_STRIDE + (static_cast<uint32_t>(q * 32) << 16);
      float swc = 0.f;
      if constexpr (I8) swc = (col < p.N && p.splits == 1) ? p.sw[col] : 0.f;
#pragma unroll 1
      for (int c = 0; c < (RB + 31) / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
        if constexpr (CLUSTER) {                        // the ring is idle: every stage has been multiplied
          uint32_t* vals = reinterpret_cast<uint32_t*>(tiles);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c * 32 + j < RB) vals[(c * 32 + j) * SK_BM + q * 32 + lane] = r[j];
        } else if (col < p.N) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int m = c * 32 + j;
            if (m < p.rows && m < RB) {
              if (p.splits == 1) {
                float v;
                if constexpr (I8) v = __fmul_rn(static_cast<float>(static_cast<int>(r[j])), __fmul_rn(p.sx[m], swc));
                else v = __uint_as_float(r[j]);
                if (p.R) v += __bfloat162float(static_cast<const __nv_bfloat16*>(p.R)[static_cast<size_t>(m) * p.ldr + col]);
                static_cast<__nv_bfloat16*>(p.C)[static_cast<size_t>(m) * p.ldc + col] = __float2bfloat16_rn(v);
              } else {
                static_cast<uint32_t*>(p.C)[(static_cast<size_t>(split) * p.rows + m) * p.N + col] = r[j];
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
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  if constexpr (CLUSTER) {
    // CTA r adds its share of the tile's (row, four columns) words over all splits, in split order
    __syncwarp();
    cluster_sync_all();
    const int c = p.splits, rank = blockIdx.y;
    const int words = p.rows * (SK_BM / 4), w1 = (rank + 1) * words / c;
    int i = rank * words / c + threadIdx.x;             // SK_THREADS is a multiple of a row's 32 words: the columns stay
    const int col4 = (i & (SK_BM / 4 - 1)) * 4, n = blockIdx.x * SK_BM + col4;
    const bool live = n < p.N;                          // N is a multiple of 8
    const __nv_bfloat16* R = static_cast<const __nv_bfloat16*>(p.R);
    __nv_bfloat16* C = static_cast<__nv_bfloat16*>(p.C);
    const bool wide = ((p.ldc | p.ldr) & 3) == 0 && ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(R)) & 7) == 0;
    float sw[4] = {0.f, 0.f, 0.f, 0.f};
    if (I8 && live) {
#pragma unroll
      for (int e = 0; e < 4; ++e) sw[e] = p.sw[n + e];
    }
    const uint32_t base = smem_u32(tiles) + col4 * 4;
#pragma unroll 2
    for (; live && i < w1; i += SK_THREADS) {
      const int m = i / (SK_BM / 4);
      float4 v[SK_MAX_CLUSTER];
#pragma unroll
      for (int s = 0; s < SK_MAX_CLUSTER; ++s)
        if (s < c) v[s] = ld_cluster_f4(mapa_shared(base + m * SK_BM * 4, s));
      float f[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
      if constexpr (I8) {
        const float sx = p.sx[m];
        int acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < SK_MAX_CLUSTER; ++s)
          if (s < c) {
            acc[0] += __float_as_int(v[s].x); acc[1] += __float_as_int(v[s].y);
            acc[2] += __float_as_int(v[s].z); acc[3] += __float_as_int(v[s].w);
          }
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = __fmul_rn(static_cast<float>(acc[e]), __fmul_rn(sx, sw[e]));
      } else {
#pragma unroll
        for (int s = 1; s < SK_MAX_CLUSTER; ++s)
          if (s < c) { f[0] += v[s].x; f[1] += v[s].y; f[2] += v[s].z; f[3] += v[s].w; }
      }
      const __nv_bfloat16* res = R ? R + static_cast<size_t>(m) * p.ldr + n : nullptr;
      __nv_bfloat16* out = C + static_cast<size_t>(m) * p.ldc + n;
      if (wide) {
        if (res) {
          const uint2 w = *reinterpret_cast<const uint2*>(res);
          f[0] += bf16_lo(w.x); f[1] += bf16_hi(w.x); f[2] += bf16_lo(w.y); f[3] += bf16_hi(w.y);
        }
        *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (res) f[e] += __bfloat162float(res[e]);
          out[e] = __float2bfloat16_rn(f[e]);
        }
      }
    }
    cluster_sync_all();                                 // nobody leaves while its sums are being read
  }
}

// C[m, n] = bf16(sum over splits in split order (+ scales) + R[m, n]). Four columns (16 bytes of every partial) per thread
// with up to eight splits' loads in flight: the partials lie in L2, and a column per thread with one load after another
// was bound by its latency. 64 rows of the three split products of an 8B layer: 4.9 -> 2.8 us each.
template <bool I8>
__global__ void __launch_bounds__(128)
skinny_reduce_kernel(const uint32_t* part, int splits, int rows, int N4, const float* sx, const float* sw,
                     const __nv_bfloat16* R, int ldr, __nv_bfloat16* C, int ldc) {
  pdl_trigger();
  pdl_wait();
  const bool wide = (reinterpret_cast<uintptr_t>(part) & 15) == 0;     // a caller's workspace may start anywhere
  const int n4 = blockIdx.x * 128 + threadIdx.x, m = blockIdx.y;
  if (n4 >= N4) return;
  const size_t plane = static_cast<size_t>(rows) * N4, at = static_cast<size_t>(m) * N4 + n4;
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  int acc[4] = {0, 0, 0, 0};
  for (int s0 = 0; s0 < splits; s0 += 8) {
    uint4 v[8];
#pragma unroll
    for (int x = 0; x < 8; ++x)
      if (s0 + x < splits) {
        const uint32_t* p = part + ((s0 + x) * plane + at) * 4;
        v[x] = wide ? *reinterpret_cast<const uint4*>(p) : make_uint4(p[0], p[1], p[2], p[3]);
      }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      if (s0 + x < splits) {
        const uint32_t w[4] = {v[x].x, v[x].y, v[x].z, v[x].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if constexpr (I8) acc[e] += static_cast<int>(w[e]);
          else f[e] = s0 + x == 0 ? __uint_as_float(w[e]) : f[e] + __uint_as_float(w[e]);
        }
      }
    }
  }
  const int n = n4 * 4;
  __nv_bfloat16* c = C + static_cast<size_t>(m) * ldc + n;
  const __nv_bfloat16* r = R ? R + static_cast<size_t>(m) * ldr + n : nullptr;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if constexpr (I8) f[e] = __fmul_rn(static_cast<float>(acc[e]), __fmul_rn(sx[m], sw[n + e]));
    if (r) f[e] += __bfloat162float(r[e]);
    c[e] = __float2bfloat16_rn(f[e]);
  }
}

// Clusters of `c` CTAs that the current device holds at once; asked for once per device and size.
template <int RB, bool I8>
static int skinny_clusters(int c) {
  auto kern = gemm_skinny_kernel<RB, I8, true>;
  static std::atomic<int> known[64][SK_MAX_CLUSTER + 1] = {};      // count + 1
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return 0;
  const bool keep = device >= 0 && device < 64;
  if (keep) {
    const int k = known[device][c].load(std::memory_order_relaxed);
    if (k > 0) return k - 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, c); cfg.blockDim = dim3(SK_THREADS); cfg.dynamicSmemBytes = SkinnyCfg<RB>::SMEM_BYTES;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = c; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
  if (keep) known[device][c].store(n + 1, std::memory_order_relaxed);
  return n;
}

// Whether the splits of `nt` column tiles finish inside the kernel; < 0: the launch cannot be prepared.
template <int RB, bool I8>
static int skinny_in_cluster(int nt, int splits) {
  if (splits < 2 || splits > SK_MAX_CLUSTER) return 0;
  static PerDeviceOnce attr;
  if (allow_smem(attr, gemm_skinny_kernel<RB, I8, true>, SkinnyCfg<RB>::SMEM_BYTES, SB_ERR_LAUNCH)) return -1;
  return nt <= skinny_clusters<RB, I8>(splits);
}

// in_cluster: set when the splits finish inside the kernel, p.C is then the output. `workspace` takes the partials otherwise.
template <int RB, bool I8>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, SkinnyParams p, void* workspace, bool* in_cluster,
                         cudaStream_t stream) {
  using Cfg = SkinnyCfg<RB>;
  const int nt = (p.N + SK_BM - 1) / SK_BM;
  auto clustered = gemm_skinny_kernel<RB, I8, true>;
  static PerDeviceOnce attr;
  const int fits = skinny_in_cluster<RB, I8>(nt, p.splits);
  if (fits < 0) return SB_ERR_LAUNCH;
  *in_cluster = fits > 0;
  if (*in_cluster)
    return launch_dep_cluster(clustered, dim3(nt, p.splits), dim3(SK_THREADS), Cfg::SMEM_BYTES, stream, p.splits, true, tw, tx,
                              p) == cudaSuccess ? 0 : SB_ERR_LAUNCH;
  auto kern = gemm_skinny_kernel<RB, I8, false>;
  if (allow_smem(attr, kern, Cfg::SMEM_BYTES, SB_ERR_LAUNCH)) return SB_ERR_LAUNCH;
  if (p.splits > 1) p.C = workspace;
  const int items = nt * p.splits;
  return launch_dep(kern, dim3(items < num_sms() ? items : num_sms()), dim3(SK_THREADS), Cfg::SMEM_BYTES, stream, tw, tx, p) ==
                 cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

// The number of k ranges that `splits` asks for (<= 0: one work item per SM), made whole; returns the k-blocks of a range.
static int skinny_split(int N, int K, int is_i8, int* splits) {
  const int bke = is_i8 ? 128 : 64;
  const int num_kb = (K + bke - 1) / bke;
  const int nt = (N + SK_BM - 1) / SK_BM;
  int s = *splits;
  if (s <= 0) {
    s = num_sms() / nt;                             // one work item per SM, no second round
    if (s < 1) s = 1;
    const int max_splits = num_kb / 4 > 0 ? num_kb / 4 : 1;      // at least four k-blocks per item
    if (s > max_splits) s = max_splits;
  }
  if (s > num_kb) s = num_kb;
  const int kbps = (num_kb + s - 1) / s;
  *splits = (num_kb + kbps - 1) / kbps;
  return kbps;
}

}  // namespace sb

using namespace sb;

// Kernels that sb_gemm_skinny launches for these sizes on the current device: 1, or 2 where split sums are added from memory.
extern "C" int sb_gemm_skinny_launches(int rows, int N, int K, int is_i8, int splits) {
  if (rows <= 0 || rows > 64 || N <= 0 || K <= 0) return 0;
  skinny_split(N, K, is_i8, &splits);
  const int nt = (N + SK_BM - 1) / SK_BM;
  const auto in_cluster = rows <= 16   ? (is_i8 ? skinny_in_cluster<16, true> : skinny_in_cluster<16, false>)
                          : rows <= 32 ? (is_i8 ? skinny_in_cluster<32, true> : skinny_in_cluster<32, false>)
                                       : (is_i8 ? skinny_in_cluster<64, true> : skinny_in_cluster<64, false>);
  return splits > 1 && in_cluster(nt, splits) <= 0 ? 2 : 1;
}

// C[rows, N] (bf16) = X . W (+ R), rows <= 64.
//   is_i8 == 0: X bf16 [rows, ldx], W bf16 [K, N] (row pitch ldw);
//   is_i8 == 1: X int8 [rows, ldx] with row scales sx, W int8 [N, K] (transposed codes, row pitch ldw, K % 16 == 0)
//               with column scales sw.
// Bases 16-byte aligned, pitches multiples of 16 bytes, N % 8 == 0. workspace: splits * rows * N 32-bit words, read
// only when the k range is split and its splits do not finish in a cluster (splits <= 0 lets the launcher fill the GPU: about one
// work item per SM).
extern "C" int sb_gemm_skinny(const void* X, int ldx, const void* W, int ldw, void* C, int ldc, const void* R, int ldr,
                              int rows, int N, int K, int is_i8, const float* sx, const float* sw, int splits,
                              void* workspace, int* status, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (rows <= 0 || rows > 64 || N <= 0 || K <= 0 || (N & 7) || !status) return SB_ERR_ARG;
  if (is_i8 && (!sx || !sw || (K & 15) || (ldx & 15) || (ldw & 15))) return SB_ERR_ARG;
  if (!is_i8 && ((ldx & 7) || (ldw & 7))) return SB_ERR_ALIGN;
  const int kbps = skinny_split(N, K, is_i8, &splits);
  if (splits > 1 && !workspace) return SB_ERR_ARG;
  const int rb = rows <= 16 ? 16 : rows <= 32 ? 32 : 64;
  CUtensorMap tw, tx;
  int rc;
  if (is_i8) {
    rc = make_tmap_2d_bf16(&tw, W, static_cast<uint64_t>(K) / 2, N, static_cast<uint64_t>(ldw) / 2, 64, SK_BM);
    if (rc) return rc;
    rc = make_tmap_2d_bf16(&tx, X, static_cast<uint64_t>(K) / 2, rows, static_cast<uint64_t>(ldx) / 2, 64, rb);
  } else {
    rc = make_tmap_2d_bf16(&tw, W, N, K, ldw, 64, 64);
    if (rc) return rc;
    rc = make_tmap_2d_bf16(&tx, X, K, rows, ldx, 64, rb);
  }
  if (rc) return rc;
  SkinnyParams p;
  p.rows = rows; p.N = N; p.K = K; p.splits = splits; p.kb_per_split = kbps;
  p.C = C; p.ldc = ldc; p.R = R; p.ldr = ldr; p.sx = sx; p.sw = sw; p.status = status;
  bool in_cluster = false;
#define SB_SKINNY(RB_)                                                                            \
  rc = is_i8 ? launch_skinny<RB_, true>(tw, tx, p, workspace, &in_cluster, stream)                \
             : launch_skinny<RB_, false>(tw, tx, p, workspace, &in_cluster, stream)
  if (rb == 16) SB_SKINNY(16); else if (rb == 32) SB_SKINNY(32); else SB_SKINNY(64);
#undef SB_SKINNY
  if (rc) return rc;
  if (splits > 1 && !in_cluster) {
    const dim3 grid_r((N / 4 + 127) / 128, rows);          // N is a multiple of 8
    auto kern = is_i8 ? skinny_reduce_kernel<true> : skinny_reduce_kernel<false>;
    if (launch_dep(kern, grid_r, dim3(128), 0, stream, static_cast<const uint32_t*>(workspace), splits, rows, N / 4, sx, sw,
                   static_cast<const __nv_bfloat16*>(R), ldr, static_cast<__nv_bfloat16*>(C), ldc) != cudaSuccess)
      return SB_ERR_LAUNCH;
  }
  return 0;
}
