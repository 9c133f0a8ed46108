// Deterministic device-side token sampler: repetition penalty -> greedy (T <= 0) or softmax(x / T)
// -> top-k -> top-p -> renormalise -> inverse-CDF draw, one cluster of CTAs per logits row, no host round trip.
//
// Policy and RNG stream follow the reference's host sampler (scirust-sciagent/src/generate.rs:202-337;
// splitmix64-seeded xorshift64, u = (s >> 11) / 2^53) and its WGSL device sampler's purpose: keep the
// token on the device. Differences by design: probabilities are turned into 32-bit fixed-point
// weights w_j = floor(exp((x_j - max) / T) * 2^32) and every sum is an integer sum, so the result does
// not depend on the order in which threads add (atomics on integers are order-free) and a seed gives
// the same tokens on every run and every grid shape. Ranking is (weight descending, id ascending),
// the host sampler's order; rank cut-offs and the draw are found with radix-select passes over the
// row instead of a sort. The host sampler adds floats sequentially, so the two can differ only when
// the uniform draw falls within rounding distance of a CDF boundary.
//
// What bounds it: a row is read once (0.5 MB at a vocabulary of 128 k) and then walked about ten times, so with one
// CTA per row the passes over global memory set the pace, whatever the number of rows. A row is spread over the
// shared memory of a cluster instead: of eight CTAs each holds 64 KB, a pass takes 16 words per thread, and the CTAs
// exchange only their 256-bin histograms (distributed shared memory, one cluster barrier per radix level, two
// histogram buffers in turn). The bin scan runs in one warp by shuffles instead of in one thread, the number of
// ties falls out of the last level, and the second walk starts from the first walk's top-level histogram. 16 rows of
// 128256 logits, top-k 50, top-p 0.95: 418 us with one CTA per row, 78 us so (147 us while all 32 warps scanned the bins
// of every level, eight neighbours to a lane and so sixteen lanes to a bank).
//
// Each of the ten levels that are left costs a barrier, an exchange and a scan, about 6 us, and mostly sorts out a few
// dozen words. So when the first level, whose histogram is made by the pass that makes the weights, leaves no more than
// SAMP_LIST words at or above the digit that the cut falls into, these go to one CTA, which ranks them and finishes alone.
// Ranks, sums and ties are those of the walks. The same 16 rows, normal logits of deviation 2.5: 26.5 us, of which half was a second
// wave for the sixteenth cluster of eight; 17.8 in clusters of four (sample_cluster). Not taken where the cut
// falls among the words below 1/256 of the largest, whose first digit is 0 (top-k without top-p on a confident row: deviation
// 8, top-k 50 73 us, with top-p 0.95 24), nor where more words than SAMP_LIST share the digit (a nucleus of 0.9 alone 79; these
// three in clusters of eight).
#include <atomic>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "api.h"
#include "per_device.h"

namespace sb {

namespace cg = cooperative_groups;

constexpr int SAMP_THREADS = 1024;
constexpr int SAMP_MAX_WINDOW = 256;
constexpr int SAMP_CLUSTER = 8;                 // portable cluster size
constexpr int SAMP_SLICE_WORDS = 48 * 1024;     // 192 KB of a CTA's shared memory; longer slices stay in `work`
// Up to here one CTA holds the row: a cluster barrier costs more than a pass over so few words.
constexpr int SAMP_SINGLE_MAX_V = 8192;
// Words that one CTA finishes: a thread compares its word with all others, 512 x 512 comparisons take about 4 us.
constexpr int SAMP_LIST = 512;

struct SampleParams {
  const float* logits; int ld; int V;
  int slice;                              // words of a row per CTA, a multiple of 4
  float temperature; int top_k; float top_p;
  float rep_penalty; int rep_window;
  const int64_t* recent; int recent_ld;   // [B, recent_ld] token history (most recent last), may be null
  const int* n_recent;                    // [B] valid entries per row
  uint64_t* rng_state;                    // [B] xorshift64 states, advanced by one draw per call
  int64_t* out_tokens;                    // [B]
  int64_t* generated; int gen_stride; int step;   // optional [B, gen_stride] log of emitted tokens
  uint32_t* work;                         // [B, V] scratch, used when a slice does not fit shared memory
};

// One CTA's histogram of a radix level. Weights are summed as two 16-bit halves in 32-bit words while a slice has at
// most 65536 words (32-bit shared atomics are native, 64-bit ones a compare-and-swap loop), else as 64-bit words.
struct SampHist {
  uint32_t cnt[256];
  union {
    struct { uint32_t lo[256], hi[256]; } half;
    unsigned long long sum[256];
  };
};

// The bins of a level over the cluster: a lane scans eight neighbours, so bin d lies at d + d / 8 (a stride of nine words
// between lanes; eight would put 16 lanes on one bank).
constexpr int SAMP_BINS = 256 + 32;
__device__ __forceinline__ int samp_bin(int d) { return d + (d >> 3); }

struct SampShared {
  SampHist h[2];
  unsigned long long tot_cnt[SAMP_BINS], tot_sum[SAMP_BINS];   // of the level being scanned, over the cluster
  unsigned long long top_cnt[SAMP_BINS], top_sum[SAMP_BINS];   // level 0
  int cut_d;                                       // result of the scan
  unsigned long long cut_cnt, cut_sum, in_cnt, in_sum;
  unsigned long long total;                        // this CTA's weight sum
  float vmax;                                      // this CTA's maximum
  float red[SAMP_THREADS / 32];
  unsigned long long red_u[SAMP_THREADS / 32];
  int64_t tok[SAMP_MAX_WINDOW];
  int n_list;                                      // rank 0's copy counts
  unsigned long long list[SAMP_LIST], ranked[SAMP_LIST];   // weight << 32 | ~id: larger is earlier in the ranking
};

template <bool SMEM>
struct Row {
  uint32_t* w;          // this CTA's slice
  int n, base;          // its length and the id of its first element

  // Visits (local index, word) of the slice, 16 bytes at a time; the slice is 16-byte aligned and padded.
  template <class F>
  __device__ __forceinline__ void each(F&& f) const {
    if constexpr (SMEM) {
      const int n4 = n >> 2;
#pragma unroll 2
      for (int j = threadIdx.x; j < n4; j += SAMP_THREADS) {
        const uint4 a = reinterpret_cast<const uint4*>(w)[j];
        f(4 * j, a.x); f(4 * j + 1, a.y); f(4 * j + 2, a.z); f(4 * j + 3, a.w);
      }
      const int j = 4 * n4 + threadIdx.x;
      if (j < n) f(j, w[j]);
    } else {
      for (int j = threadIdx.x; j < n; j += SAMP_THREADS) f(j, w[j]);
    }
  }
};

template <bool SMEM>
__device__ __forceinline__ void hist_add(SampHist& h, int d, uint32_t c, unsigned long long s, uint32_t lo, uint32_t hi) {
  atomicAdd(&h.cnt[d], c);
  if constexpr (SMEM) { atomicAdd(&h.half.lo[d], lo); atomicAdd(&h.half.hi[d], hi); }
  else atomicAdd(&h.sum[d], s);
}

// A thread batches the run of equal digits it sees: near-uniform rows put everything into one bin. Digit 0 is not added.
template <bool SMEM>
struct RunOfDigits {
  SampHist& h;
  int cur = 0;
  uint32_t c = 0, lo = 0, hi = 0;
  unsigned long long s = 0;
  __device__ __forceinline__ void flush() {
    if (c) hist_add<SMEM>(h, cur, c, s, lo, hi);
  }
  __device__ __forceinline__ void add(int d, uint32_t v) {
    if (d != cur) { flush(); cur = d; c = 0; s = 0; lo = 0; hi = 0; }
    c += 1;
    if constexpr (SMEM) { lo += v & 0xffffu; hi += v >> 16; }
    else s += v;
  }
};

// Sums the cluster's histograms into tot_cnt / tot_sum (bin 0, usually the fullest, is not counted: the scan gets it from
// the totals) and clears the buffer of the next level.
template <bool SMEM>
__device__ void combine(cg::cluster_group& cl, SampShared& s, int buf) {
  cl.sync();
  const int t = threadIdx.x;
  if (t < 256) {
    unsigned long long c = 0, v = 0;
    const int nr = cl.num_blocks();
#pragma unroll
    for (int r = 0; r < SAMP_CLUSTER; ++r) {       // all remote loads in flight at once
      if (r < nr) {
        const SampHist* h = cl.map_shared_rank(&s.h[buf], r);
        c += h->cnt[t];
        if constexpr (SMEM) v += (static_cast<unsigned long long>(h->half.hi[t]) << 16) + h->half.lo[t];
        else v += h->sum[t];
      }
    }
    s.tot_cnt[samp_bin(t)] = c;
    s.tot_sum[samp_bin(t)] = v;
  } else if (t < 512) {
    // every CTA has read this buffer's previous level before it arrived at the barrier above
    SampHist& h = s.h[buf ^ 1];
    h.cnt[t - 256] = 0;
    h.sum[t - 256] = 0;
  }
  __syncthreads();
}

// The first digit, from 255 down, where the running count reaches limit_count or the running sum reaches target
// (passes it when `strict`); digit 0 when none above does. Warp 0 scans, eight bins per lane, all loads first; the
// digit, the counts and sums of everything above it and its own go to s.cut_* and s.in_*. in_cnt / in_sum: totals over
// the 256 bins.
__device__ void scan_bins(SampShared& s, const unsigned long long* cnt, const unsigned long long* sum,
                          unsigned long long in_cnt, unsigned long long in_sum, unsigned long long cnt_before,
                          unsigned long long sum_before, unsigned long long limit_count, unsigned long long target,
                          bool strict) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int hi = 255 - 8 * lane;                 // this lane's bins: hi, hi - 1, ... hi - 7
    unsigned long long cb[8], sb_[8], c8 = 0, s8 = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { cb[i] = cnt[samp_bin(hi - i)]; sb_[i] = sum[samp_bin(hi - i)]; }
    if (lane == 31) cb[7] = sb_[7] = 0;            // bin 0 is set below
#pragma unroll
    for (int i = 0; i < 8; ++i) { c8 += cb[i]; s8 += sb_[i]; }
    unsigned long long c = c8, v = s8;             // inclusive over lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long pc = __shfl_up_sync(0xffffffffu, c, o), ps = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) { c += pc; v += ps; }
    }
    if (lane == 31) { cb[7] = in_cnt - c; sb_[7] = in_sum - v; }
    c += cnt_before - c8;
    v += sum_before - s8;                          // before this lane's first bin
    int d = 0;
    unsigned long long kc = c, ks = v, kic = 0, kis = 0;
    bool found = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long ci = c + cb[i], si = v + sb_[i];
      if (!found && ((cb[i] != 0 && (ci >= limit_count || (strict ? si > target : si >= target))) || hi - i == 0)) {
        found = true;
        d = hi - i; kc = c; ks = v; kic = cb[i]; kis = sb_[i];
      }
      c = ci; v = si;
    }
    if (lane == __ffs(__ballot_sync(0xffffffffu, found)) - 1) {     // lane 31 always finds bin 0
      s.cut_d = d; s.cut_cnt = kc; s.cut_sum = ks; s.in_cnt = kic; s.in_sum = kis;
    }
  }
  __syncthreads();
}

struct Walk {                   // result of one ranked walk
  unsigned long long sum;       // inclusive weight sum where the walk stopped
  unsigned long long take, ties;// the stopping element is the take-th of `ties` elements of this weight
  uint32_t weight;
};

// Ranked walk over the weights of one row (rank = weight descending, id ascending). Stops at the
// first rank r where either r + 1 == limit_count, or the inclusive sum reaches `target`
// (>= target, or > target when `strict`). `buf` is the histogram buffer to use next (clear on entry and on exit).
template <bool SMEM>
__device__ Walk ranked_walk(cg::cluster_group& cl, SampShared& s, const Row<SMEM>& row, int& buf,
                            unsigned long long n, unsigned long long z, unsigned long long limit_count,
                            unsigned long long target, bool strict) {
  uint32_t prefix = 0;
  unsigned long long cnt_before = 0, sum_before = 0, in_cnt = n, in_sum = z;   // in_*: of the elements under `prefix`
#pragma unroll 1
  for (int level = 0; level < 4; ++level) {
    const int shift = 24 - 8 * level;
    const unsigned long long *tc = s.tot_cnt, *ts = s.tot_sum;
    if (level == 0) {
      tc = s.top_cnt; ts = s.top_sum;
    } else {
      const uint32_t mask_hi = 0xffffffffu << (shift + 8);
      SampHist& h = s.h[buf];
      RunOfDigits<SMEM> run{h};
      row.each([&](int, uint32_t v) {
        const int d = (v >> shift) & 0xff;
        if ((v & mask_hi) == prefix && d != 0) run.add(d, v);
      });
      run.flush();
      combine<SMEM>(cl, s, buf);
      buf ^= 1;
    }
    scan_bins(s, tc, ts, in_cnt, in_sum, cnt_before, sum_before, limit_count, target, strict);
    prefix |= static_cast<uint32_t>(s.cut_d) << shift;
    in_cnt = s.in_cnt;
    in_sum = s.in_sum;
    cnt_before = s.cut_cnt;
    sum_before = s.cut_sum;
    __syncthreads();                               // all have read the cut
  }
  // all elements with weight == prefix are tied; they are taken in id order
  const unsigned long long v = prefix;
  Walk out;
  out.weight = prefix;
  out.ties = in_cnt;
  unsigned long long take = in_cnt;                    // ties consumed, the stopping element included
  if (limit_count - cnt_before < take) take = limit_count - cnt_before;
  if (v > 0) {
    unsigned long long need;                            // ties needed for the sum criterion
    if (strict) need = target >= sum_before ? (target - sum_before) / v + 1 : 1;
    else need = target > sum_before ? (target - sum_before - 1) / v + 1 : 1;   // rounded up; target may be ~0
    if (need < take) take = need;
  }
  if (take < 1) take = 1;
  out.take = take;
  out.sum = sum_before + take * v;
  return out;
}

// The cumulative probability's target in weight units, never below one.
__device__ __forceinline__ unsigned long long nucleus_target(float top_p, unsigned long long z) {
  const double d = static_cast<double>(top_p) * static_cast<double>(z);
  return d <= 1.0 ? 1ull : static_cast<unsigned long long>(ceil(d));
}
// Where the draw falls in a kept sum of zz; advances the row's generator.
__device__ __forceinline__ unsigned long long draw_target(uint64_t& st, unsigned long long zz) {
  st ^= st << 13; st ^= st >> 7; st ^= st << 17;
  const float u = static_cast<float>(static_cast<double>(st >> 11) / 9007199254740992.0);
  unsigned long long target = static_cast<unsigned long long>(static_cast<double>(u) * static_cast<double>(zz));
  if (zz > 0 && target >= zz) target = zz - 1;
  return target;
}

// One CTA finishes the row: s.list holds every word down to the first digit of the cut (n of them, all above zero). The
// kept set ends at the first rank r with r + 1 == limit or an inclusive sum of at least tp; the draw takes the first rank
// whose inclusive sum is above its target. Returns the id to the thread that holds it, -1 to the others.
__device__ int finish_list(SampShared& s, int n, unsigned long long limit, unsigned long long tp, bool cut,
                           unsigned long long z, uint64_t& st) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t < n) {
    const unsigned long long mine = s.list[t];
    int r = 0;
#pragma unroll 8
    for (int k = 0; k < n; ++k) r += s.list[k] > mine;       // ids differ, so no two words are equal
    s.ranked[r] = mine;
  }
  __syncthreads();
  const unsigned long long key = t < n ? s.ranked[t] : 0;
  unsigned long long sum = key >> 32;                        // inclusive over ranks
  if (t < SAMP_LIST) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) s.red_u[warp] = sum;
  }
  __syncthreads();
  if (t < SAMP_LIST) {
    for (int k = 0; k < warp; ++k) sum += s.red_u[k];
    const unsigned long long before = sum - (key >> 32);
    // exactly one rank is the first to reach the limit or the sum
    const unsigned long long place = static_cast<unsigned long long>(t) + 1;
    if (t < n && (place == limit || sum >= tp) && place <= limit && before < tp) s.cut_sum = sum;
  }
  __syncthreads();
  const unsigned long long zz = cut ? s.cut_sum : z;
  const unsigned long long target = draw_target(st, zz);
  const bool hit = t < n && sum > target && sum - (key >> 32) <= target;
  return hit ? static_cast<int>(~static_cast<uint32_t>(key)) : -1;
}

template <bool SMEM>
__global__ void __launch_bounds__(SAMP_THREADS, 1)
sample_rows_kernel(const SampleParams p) {
  extern __shared__ __align__(16) uint32_t slice_smem[];
  __shared__ SampShared s;
  cg::cluster_group cl = cg::this_cluster();
  const int nr = cl.num_blocks(), rank = cl.block_rank();
  const int row_id = blockIdx.x / nr;
  const int V = p.V, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const float* x = p.logits + static_cast<size_t>(row_id) * p.ld;
  Row<SMEM> row;
  row.base = rank * p.slice;
  row.n = max(0, min(p.slice, V - row.base));
  row.w = SMEM ? slice_smem : p.work + static_cast<size_t>(row_id) * V + min(row.base, V);
  float* wf = reinterpret_cast<float*>(row.w);
  uint64_t st = p.rng_state[row_id];          // on its way long before the draw

  // ---- penalised copy of the slice ----
  const float* xs = x + min(row.base, V);
  float mx = -INFINITY;
  if (SMEM && (reinterpret_cast<uintptr_t>(xs) & 15) == 0) {
    const int n4 = row.n >> 2;
#pragma unroll 4
    for (int j = t; j < n4; j += SAMP_THREADS) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(xs) + j);
      reinterpret_cast<float4*>(wf)[j] = a;
      mx = fmaxf(fmaxf(mx, fmaxf(a.x, a.y)), fmaxf(a.z, a.w));
    }
    const int j = 4 * n4 + t;
    if (j < row.n) { wf[j] = xs[j]; mx = fmaxf(mx, xs[j]); }
  } else {
#pragma unroll 4
    for (int j = t; j < row.n; j += SAMP_THREADS) { const float a = xs[j]; wf[j] = a; mx = fmaxf(mx, a); }
  }
  if (t < 512) {
    s.h[t >> 8].cnt[t & 255] = 0;
    s.h[t >> 8].sum[t & 255] = 0;
  }
  if (t == 0) s.n_list = 0;
  int n_win = 0;
  if (p.rep_penalty > 1.0f && p.recent && p.n_recent) {
    const int n = p.n_recent[row_id];
    n_win = min(min(n, p.rep_window), SAMP_MAX_WINDOW);
    const int64_t* rec = p.recent + static_cast<size_t>(row_id) * p.recent_ld + (n - n_win);
    if (t < n_win) s.tok[t] = rec[t];
  }
  __syncthreads();
  if (t < n_win) {
    // every occurrence in the window applies the penalty once more; the first occurrence's thread applies them all
    const int64_t tk = s.tok[t];
    const int64_t at = tk - row.base;
    if (tk >= 0 && tk < V && at >= 0 && at < row.n) {
      bool first = true;
      int times = 0;
      for (int k = 0; k < n_win; ++k) {
        if (s.tok[k] != tk) continue;
        if (k < t) { first = false; break; }
        ++times;
      }
      if (first) {
        float l = wf[at];
        for (int k = 0; k < times; ++k) l = l > 0.f ? l / p.rep_penalty : l * p.rep_penalty;
        wf[at] = l;
      }
    }
  }
  __syncthreads();

  int token = -1;              // known to the thread that writes it out
  if (n_win > 0) {             // the penalty may have taken the maximum
    mx = -INFINITY;
    for (int j = t; j < row.n; j += SAMP_THREADS) mx = fmaxf(mx, wf[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) s.red[warp] = mx;
  __syncthreads();
  if (warp == 0) {
    mx = s.red[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) s.vmax = mx;
  }
  cl.sync();
  // a lane per CTA: one trip to the others' memory instead of eight in a row
  mx = *cl.map_shared_rank(&s.vmax, lane < nr ? lane : rank);
#pragma unroll
  for (int o = SAMP_CLUSTER / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  mx = __shfl_sync(0xffffffffu, mx, 0);
  // fixed-point weights, their total and the first level's histogram
  unsigned long long local = 0;
  const float inv_t = 1.0f / p.temperature;
  {
    RunOfDigits<SMEM> run{s.h[0]};
    auto weigh = [&](float l) {
      const float e = expf((l - mx) * inv_t);                // in [0, 1]
      const float f = e * 4294967296.0f;
      const uint32_t q = f >= 4294967040.0f ? 0xffffffffu : static_cast<uint32_t>(f);
      local += q;
      if (q >> 24) run.add(q >> 24, q);
      return q;
    };
    if constexpr (SMEM) {
      const int n4 = row.n >> 2;
#pragma unroll 2
      for (int j = t; j < n4; j += SAMP_THREADS) {
        const float4 a = reinterpret_cast<const float4*>(wf)[j];
        reinterpret_cast<uint4*>(row.w)[j] = make_uint4(weigh(a.x), weigh(a.y), weigh(a.z), weigh(a.w));
      }
      const int j = 4 * n4 + t;
      if (j < row.n) row.w[j] = weigh(wf[j]);
    } else {
      for (int j = t; j < row.n; j += SAMP_THREADS) row.w[j] = weigh(wf[j]);
    }
    run.flush();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if (lane == 0) s.red_u[warp] = local;
  __syncthreads();
  if (warp == 0) {
    local = s.red_u[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0) s.total = local;
  }
  combine<SMEM>(cl, s, 0);
  int buf = 1;
  unsigned long long z = lane < nr ? *cl.map_shared_rank(&s.total, lane) : 0;
#pragma unroll
  for (int o = SAMP_CLUSTER / 2; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  z = __shfl_sync(0xffffffffu, z, 0);
  if (t < SAMP_BINS) { s.top_cnt[t] = s.tot_cnt[t]; s.top_sum[t] = s.tot_sum[t]; }
  // kept set: first min(top_k, V) ranks, cut where the cumulative probability reaches top_p
  const unsigned long long n_all = static_cast<unsigned long long>(V);
  const unsigned long long limit = (p.top_k > 0 && p.top_k < V) ? static_cast<unsigned long long>(p.top_k) : n_all;
  const bool cut = limit < n_all || p.top_p < 1.0f;
  const unsigned long long tp = p.top_p < 1.0f ? nucleus_target(p.top_p, z) : ~0ull;   // ~0: only the count stops the walk
  {
    // the first level of the first walk: the cut's, or the draw's when everything is kept
    uint64_t peek = st;
    const unsigned long long target = cut ? tp : draw_target(peek, z);
    scan_bins(s, s.tot_cnt, s.tot_sum, n_all, z, 0, 0, limit, target, !cut);
    const uint32_t d0 = static_cast<uint32_t>(s.cut_d);
    const unsigned long long n_up = s.cut_cnt + s.in_cnt;
    if (d0 > 0 && n_up <= SAMP_LIST) {
      SampShared* first = cl.map_shared_rank(&s, 0);
      row.each([&](int j, uint32_t v) {
        if (v >> 24 >= d0)
          first->list[atomicAdd(&first->n_list, 1)] =
              static_cast<unsigned long long>(v) << 32 | static_cast<uint32_t>(~static_cast<uint32_t>(row.base + j));
      });
      cl.sync();               // the list is whole; nobody reads another CTA's memory from here on
      if (rank != 0) return;
      token = finish_list(s, static_cast<int>(n_up), limit, tp, cut, z, st);
      if (t == 0) p.rng_state[row_id] = st;
      if (token >= 0) {
        p.out_tokens[row_id] = token;
        if (p.generated) p.generated[static_cast<size_t>(row_id) * p.gen_stride + p.step] = token;
      }
      return;
    }
    __syncthreads();           // all have read the cut
  }
  unsigned long long zz = z;
  if (cut) zz = ranked_walk<SMEM>(cl, s, row, buf, n_all, z, limit, tp, false).sum;
  // one uniform draw; every thread computes it, one stores the state after all have read it
  const unsigned long long target = draw_target(st, zz);
  const Walk wk = ranked_walk<SMEM>(cl, s, row, buf, n_all, z, n_all, target, true);
  cl.sync();
  if (rank == 0 && t == 0) p.rng_state[row_id] = st;
  if (wk.ties == 1) {
    row.each([&](int j, uint32_t v) { if (v == wk.weight) token = row.base + j; });
  } else {
    // id of the take-th smallest id among the ties: radix-select on the id (three 8-bit levels)
    unsigned long long k = wk.take - 1;   // 0-based index among ties
    uint32_t id_prefix = 0;
#pragma unroll 1
    for (int level = 0; level < 3; ++level) {
      const int shift = 16 - 8 * level;
      const uint32_t mask_hi = level == 0 ? 0u : (0xffffffffu << (shift + 8));
      row.each([&](int j, uint32_t v) {
        const uint32_t id = static_cast<uint32_t>(row.base + j);
        if (v == wk.weight && (id & mask_hi) == id_prefix) atomicAdd(&s.h[buf].cnt[(id >> shift) & 0xff], 1u);
      });
      cl.sync();
      if (t < 256) {
        unsigned long long c = 0;
        for (int r = 0; r < nr; ++r) c += cl.map_shared_rank(&s.h[buf], r)->cnt[t];
        s.tot_cnt[t] = c;
      } else if (t < 512) {
        s.h[buf ^ 1].cnt[t - 256] = 0;
      }
      buf ^= 1;
      __syncthreads();
      int d = 0;
      for (; d < 255; ++d) {
        if (k < s.tot_cnt[d]) break;
        k -= s.tot_cnt[d];
      }
      id_prefix |= static_cast<uint32_t>(d) << shift;
    }
    if (rank == 0 && t == 0) token = static_cast<int>(id_prefix);
  }
  if (token >= 0) {
    p.out_tokens[row_id] = token;
    if (p.generated) p.generated[static_cast<size_t>(row_id) * p.gen_stride + p.step] = token;
  }
  cl.sync();   // no CTA leaves while another may still read its shared memory
}

// Greedy rows (T <= 0) need one pass: the logits are read once, straight from memory, by as many CTAs of a cluster as leave
// each at least 4096 words and the grid within the GPU (a cluster of eight for every row from 8193 words on took 18.6 us
// for 64 rows of 9000, where one CTA per row takes 5.2). The ids of the penalty's window are worked out first, one thread
// each, and skipped by the pass: it looks an id up only where its logit would win, in a bitmap of the slice (of
// its low 16 bits, and then the window itself, for slices longer than that).
constexpr int SAMP_BITMAP = 65536;
constexpr int SAMP_SMALL_V = 2048, SAMP_SMALL_THREADS = 256;   // a small block starts sooner; it has a thread per id of the window
static_assert(SAMP_SMALL_THREADS >= SAMP_MAX_WINDOW, "a thread per id of the window");

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
greedy_rows_kernel(const SampleParams p) {
  __shared__ __align__(16) int tok[SAMP_MAX_WINDOW];          // -1: no id of this row
  __shared__ uint32_t bitmap[SAMP_BITMAP / 32];
  __shared__ float red[THREADS / 32];
  __shared__ int red_i[THREADS / 32];
  __shared__ float vmax;
  __shared__ int vid;
  cg::cluster_group cl = cg::this_cluster();
  const int nr = cl.num_blocks(), rank = cl.block_rank();
  const int row_id = blockIdx.x / nr;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const float* x = p.logits + static_cast<size_t>(row_id) * p.ld;
  const int base = rank * p.slice, n = max(0, min(p.slice, p.V - base));
  const float x0 = rank == 0 && t == 0 ? x[0] : 0.f;     // asked for now, looked at in the end
  // the larger value, the lower id among equals; a NaN never wins against a number
  float best = -INFINITY;
  int bi = 0x7fffffff;
  auto better = [](float ob, int oi, float b, int i) { return ob > b || (!(b > ob) && oi < i); };
  auto number = [](float v) { return v != v ? -INFINITY : v; };
  int n_win = 0;
  if (p.rep_penalty > 1.0f && p.recent && p.n_recent) {
    const int nrec = p.n_recent[row_id];
    n_win = min(min(nrec, p.rep_window), SAMP_MAX_WINDOW);
    const int64_t* rec = p.recent + static_cast<size_t>(row_id) * p.recent_ld + (nrec - n_win);
    for (int j = t; j < (min(n, SAMP_BITMAP) + 31) / 32; j += THREADS) bitmap[j] = 0;
    if (t < SAMP_MAX_WINDOW) {
      const int64_t id = t < n_win ? rec[t] : -1;
      tok[t] = id >= 0 && id < p.V ? static_cast<int>(id) : -1;
    }
    __syncthreads();
    const int tk = t < n_win ? tok[t] : -1, at = tk - base;
    if (tk >= 0 && at >= 0 && at < n) {
      const uint32_t bit = static_cast<uint32_t>(at) & (SAMP_BITMAP - 1);
      atomicOr(&bitmap[bit >> 5], 1u << (bit & 31));
      // every occurrence in the window applies the penalty once more; the first occurrence's thread applies them all
      int before = 0, times = 0;
      for (int k = 0; k < n_win; k += 4) {
        const int4 o = *reinterpret_cast<const int4*>(tok + k);
        times += (o.x == tk) + (o.y == tk) + (o.z == tk) + (o.w == tk);
        before += (o.x == tk && k < t) + (o.y == tk && k + 1 < t) + (o.z == tk && k + 2 < t) + (o.w == tk && k + 3 < t);
      }
      if (before == 0) {
        float l = x[tk];
        for (int k = 0; k < times; ++k) l = l > 0.f ? l / p.rep_penalty : l * p.rep_penalty;
        best = number(l);
        bi = tk;
      }
    }
    __syncthreads();
  }

  auto visit = [&](int j, float v) {
    v = number(v);
    if (!better(v, base + j, best, bi)) return;
    if (n_win > 0) {
      const uint32_t bit = static_cast<uint32_t>(j) & (SAMP_BITMAP - 1);
      if (bitmap[bit >> 5] >> (bit & 31) & 1u) {
        bool in = n <= SAMP_BITMAP;
        for (int k = 0; k < n_win && !in; ++k) in = tok[k] == base + j;
        if (in) return;
      }
    }
    best = v;
    bi = base + j;
  };
  const float* xs = x + min(base, p.V);
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(xs) & 15) == 0) {
    const int n4 = n >> 2;
    constexpr int U = 4;                       // 16-byte loads in flight
    for (int j0 = t; j0 < n4; j0 += U * THREADS) {
      float4 a[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int j = j0 + i * THREADS;
        a[i] = j < n4 ? __ldg(reinterpret_cast<const float4*>(xs) + j) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      }
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int j = j0 + i * THREADS;
        if (j >= n4 || fmaxf(fmaxf(a[i].x, a[i].y), fmaxf(a[i].z, a[i].w)) < best) continue;
        visit(4 * j, a[i].x); visit(4 * j + 1, a[i].y); visit(4 * j + 2, a[i].z); visit(4 * j + 3, a[i].w);
      }
    }
    done = 4 * n4;
  }
#pragma unroll 4
  for (int j = done + t; j < n; j += THREADS) visit(j, xs[j]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (better(ob, oi, best, bi)) { best = ob; bi = oi; }
  }
  if (lane == 0) { red[warp] = best; red_i[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    best = lane < THREADS / 32 ? red[lane] : -INFINITY;
    bi = lane < THREADS / 32 ? red_i[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ob, oi, best, bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { vmax = best; vid = bi; }
  }
  if (nr > 1) cl.sync();
  if (rank == 0 && t == 0) {
    for (int r = 1; r < nr; ++r) {
      const float ob = *cl.map_shared_rank(&vmax, r);
      const int oi = *cl.map_shared_rank(&vid, r);
      if (better(ob, oi, best, bi)) { best = ob; bi = oi; }
    }
    // the host rule starts from element 0, so a NaN there is never displaced
    const int token = (bi == 0x7fffffff || x0 != x0) ? 0 : bi;
    p.out_tokens[row_id] = token;
    if (p.generated) p.generated[static_cast<size_t>(row_id) * p.gen_stride + p.step] = token;
  }
  if (nr > 1) cl.sync();   // no CTA leaves while another may still read its shared memory
}

static int launch_clusters(void (*kern)(const SampleParams), const SampleParams& p, int rows, int cluster, int threads,
                           size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * cluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 1 : 0;      // a plain launch is a cluster of one
  return cudaLaunchKernelEx(&cfg, kern, p) == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

int num_sms();   // gemm_tcgen05.cu

static int launch_greedy(SampleParams p, int rows, cudaStream_t stream) {
  // a cluster's CTAs lie in one part of the GPU: sixteen clusters of eight do not run at once (16 rows of 128256: 12.9 us, in
  // clusters of four 7.7), so those fill three quarters of the SMs at most
  int cluster = 1;
  while (cluster < SAMP_CLUSTER && p.V / (2 * cluster) >= 4096 &&
         rows * 2 * cluster <= (cluster < 4 ? num_sms() : num_sms() * 3 / 4)) cluster *= 2;
  p.slice = ((p.V + cluster - 1) / cluster + 3) / 4 * 4;
  if (p.V <= SAMP_SMALL_V)
    return launch_clusters(greedy_rows_kernel<SAMP_SMALL_THREADS>, p, rows, cluster, SAMP_SMALL_THREADS, 0, stream);
  return launch_clusters(greedy_rows_kernel<SAMP_THREADS>, p, rows, cluster, SAMP_THREADS, 0, stream);
}

// Clusters of `c` CTAs of the sampler that the current device holds at once; asked for once per device and size.
static int sample_clusters(int c) {
  static std::atomic<int> known[64][SAMP_CLUSTER + 1] = {};
  int device = 0;
  const bool keep = cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < 64;
  if (keep) {
    const int k = known[device][c].load(std::memory_order_relaxed);
    if (k > 0) return k;
  }
  auto kern = sample_rows_kernel<true>;
  int n = num_sms() / c;
  if (c > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(SAMP_THREADS);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); n = num_sms() * 3 / 4 / c; }
  }
  if (n < 1) n = 1;
  if (keep) known[device][c].store(n, std::memory_order_relaxed);
  return n;
}

// CTAs of a row. Eight while the clusters of all rows run at once; a cluster lies in one part of the GPU, which holds 15 of eight, 33
// of four, 74 of two. Beyond that the size whose waves take least: a wave is about FIXED + the words of a slice, in half cycles, which is a
// line through the times of rows that finish by the list. 128256 logits, us, clusters of eight / four: 15 rows 16.5 / 18.5, 16 rows 25.9
// / 18.5, 64 rows 73.8 / 55.5; 32000, 64 rows, eight / four / two / one: 47.2 / 22.6 / 14.4 / 16.4. Rows that walk pay a word about five
// times over, which no size of the call tells. Over 825 calls (15 vocabularies of 8200 to 256000, 16 to 200 rows, five settings) the
// choice is 0.6 % off the best size on average, by more than 10 % in 20 (at most 22 %, 48 rows of 65536), and slower than always eight in
// five (16 rows of 151936 and 175000 that walk, 44 / 38), faster in 707.
static int sample_cluster(int V, int rows) {
  if (V <= SAMP_SINGLE_MAX_V) return 1;
  int best = SAMP_CLUSTER;
  if (rows <= sample_clusters(SAMP_CLUSTER)) return best;
  constexpr long long FIXED[4] = {20000, 25000, 27000, 28000};       // of one, two, four and eight CTAs
  long long least = 0;
  for (int k = 3, c = SAMP_CLUSTER; k >= 0; --k, c >>= 1) {
    const int words = (V + c - 1) / c, held = sample_clusters(c);
    if (c < SAMP_CLUSTER && (words + 3) / 4 * 4 > SAMP_SLICE_WORDS) break;
    const long long cost = static_cast<long long>((rows + held - 1) / held) * (FIXED[k] + words);
    if (c == SAMP_CLUSTER || cost < least) { least = cost; best = c; }
  }
  return best;
}

template <bool SMEM>
static int launch_sample(const SampleParams& p, int rows, int cluster, cudaStream_t stream) {
  auto kern = sample_rows_kernel<SMEM>;
  static PerDeviceOnce attr;
  if (SMEM && allow_smem(attr, kern, SAMP_SLICE_WORDS * 4, SB_ERR_LAUNCH)) return SB_ERR_LAUNCH;
  return launch_clusters(kern, p, rows, cluster, SAMP_THREADS, SMEM ? static_cast<size_t>(p.slice) * 4 : 0, stream);
}

}  // namespace sb

using namespace sb;

// logits: fp32 [rows, ld]; work: rows*V 32-bit words of scratch; rng_state: one xorshift64 state per
// row (advanced by one draw when temperature > 0); recent/n_recent: optional token history for the
// repetition penalty (window <= 256). vocab < 2^24.
extern "C" int sb_sample_rows(const float* logits, int ld, int rows, int V, float temperature, int top_k, float top_p,
                              float rep_penalty, int rep_window, const int64_t* recent, int recent_ld,
                              const int* n_recent, uint64_t* rng_state, int64_t* out_tokens, int64_t* generated,
                              int gen_stride, int step, uint32_t* work, void* stream) {
  if (rows <= 0 || V <= 0 || V >= (1 << 24) || !work || !out_tokens) return SB_ERR_ARG;
  if (temperature > 0.f && !rng_state) return SB_ERR_ARG;
  SampleParams p;
  p.logits = logits; p.ld = ld; p.V = V; p.temperature = temperature; p.top_k = top_k; p.top_p = top_p;
  p.rep_penalty = rep_penalty; p.rep_window = rep_window; p.recent = recent; p.recent_ld = recent_ld;
  p.n_recent = n_recent; p.rng_state = rng_state; p.out_tokens = out_tokens; p.generated = generated;
  p.gen_stride = gen_stride; p.step = step; p.work = work;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (temperature <= 0.f) return launch_greedy(p, rows, st);
  const int cluster = sample_cluster(V, rows);
  p.slice = ((V + cluster - 1) / cluster + 3) / 4 * 4;
  return p.slice <= SAMP_SLICE_WORDS ? launch_sample<true>(p, rows, cluster, st) : launch_sample<false>(p, rows, cluster, st);
}
