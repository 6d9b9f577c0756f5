// Key-to-centroid assignment on the 5th-generation tensor cores (cache_hub/kmeans.py:7-79 is the reference
// kernel): scores <k_t, x_c> for 256 tokens x all centroids of a group per CTA as tcgen05 MMAs with the
// accumulators in tensor memory, and a running top-2 per token in the epilogue.
//
//   warp 0        TMA producer: an item's two 128-token tiles, two items deep, and its group's 128-centroid tiles into a
//                 3-stage ring
//   warp 1        MMA issuer: for every centroid tile, S_a = tokens_a x centroids^T (M128 N128 K16 x D/16) for the
//                 two token tiles a = 0, 1 in turn; owns the 512 TMEM columns (two 128-column accumulators per token tile)
//   warps 2..5    epilogue of token tile 0, warps 6..9 of token tile 1: one token per thread (a TMEM lane)
// The epilogue warps scan one accumulator while the tensor core fills the other; every centroid tile staged in shared memory
// is used by both token tiles, which halves the L2 traffic per flop.  The scan bounds it: five minima and maxima per two
// scores on a pipe that takes one in two clocks.  A score's column is put into it on the FMA pipe, which is otherwise idle:
// scaled to +-500000 and rounded to a whole number by adding 1.5 * 2^23, then the column added as 32nds (6.2 clocks per score
// and scheduler; with the column in the low bits by (bits & ~31) | column, two logic operations on the pipe of the minima, 9.5).
// 8 x 65536 keys, 1024 centroids: 215 us with the logic operations, 179 with one of them (LOP3), 165 like this, 109 with the
// scan left out, and 84 at the measured matrix rate.  A CTA (one per SM) walks several 256-token items: with one item per CTA
// the start-up of each (tensor memory, barriers, the first tiles) lay open (268 us).
//
// Exactness: the fp32 tensor-core score is not the exact inner product, so a token whose best and second-best
// scores are closer than a bound on that error is put on a list and re-scored in fp64 by kmeans_recheck_list_kernel
// (exact products, index-order sum, lowest index on ties): the final assignment is the exact argmax.  The bound is a
// product of norms; where one of them is too small for an fp32 square there is no bound and every centroid is re-scored.
#pragma once
#include <cuda.h>

#include "kmeans.cuh"
#include "ptx.cuh"

namespace sq {

constexpr int kKtTokens = 256;    // tokens per CTA (two M = 128 tiles)
constexpr int kKtCent = 128;      // centroids per MMA group (N)
constexpr int kKtStages = 3;
// |tensor-core fp32 sum - exact| is bounded by (terms * 2^-22) * sum|terms| <= 2^-15 |k||x| for 128 terms; the two
// scores that are compared each carry it, and the factor of two on top covers an accumulator that truncates
constexpr float kKtTol = 1.25e-4f;
// The scan compares scores in units of |k| max|x| / kKtScale, rounded to whole ones (below 2^19, so that 32nds beside them are
// exact).  Two scores that are kKtTol |k| max|x| apart differ by kKtTol * kKtScale = 62.5 there, less two roundings of a half
// and 31/32 of column; the rest covers the rounding of the scale itself.
constexpr float kKtScale = 500000.0f;
constexpr float kKtGap = 64.6f;
// Squared norms from here on (2^-100) bound the error as stated: squares and products that underflow are below 2^-126 each,
// less than 2^-119 in all, where the bound is at least 1.25e-4 * 2^-100 = 2^-113.
constexpr float kKtMinNorm2 = 7.888609e-31f;

struct KmeansTcParams {
  int* idx;                 // [G, T]
  int* flagged;             // [cap] packed g * T + t of tokens to re-score
  int* flagged_count;       // number of entries (may exceed cap: the overflow is re-scored by a full sweep)
  int flagged_cap;
  const float* max_cnorm2;  // [G] largest squared centroid norm of the group
  int groups, num_tokens, num_centroids, bf16;
};

template <int D>
struct KmeansTcSmem {
  static constexpr int kABytes = 128 * D * 2;
  static constexpr int kBBytes = kKtCent * D * 2;
  static constexpr int kAOff = 0;
  static constexpr int kBOff = 4 * kABytes;
  static constexpr int kBarOff = kBOff + kKtStages * kBBytes;
  // a_full[2], a_empty[2], b_full[3], b_empty[3], s_full[2][2] (token tile, accumulator), s_empty[2][2]
  static constexpr int kMiscOff = kBarOff + 8 * (4 + 2 * kKtStages + 8);
  static constexpr int kTotal = kMiscOff + 16;
};

// max over the centroids of a group of sum_d x_d^2 (fp32); out is zeroed by the caller, and floats that are not negative
// order like their bits.  D / 8 lanes per row, kCnormParts CTAs per group (one read its centroids row by row: 13 us).
constexpr int kCnormParts = 8;
template <int D, bool BF16>
__global__ void __launch_bounds__(256) kmeans_cnorm_max_kernel(const uint8_t* cent, int num_centroids, float* out) {
  constexpr int kLanes = D / 8, kRows = 256 / kLanes;
  const int g = blockIdx.x, c0 = blockIdx.y * kRows + threadIdx.x / kLanes, ch = threadIdx.x % kLanes;
  const uint8_t* cg = cent + static_cast<long long>(g) * num_centroids * D * 2 + ch * 16;
  float m = 0.f;
  for (int c = c0; c < num_centroids; c += kCnormParts * kRows) {
    float f[8], s = 0.f;
    unpack8<BF16>(*reinterpret_cast<const uint4*>(cg + static_cast<long long>(c) * D * 2), f);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += f[i] * f[i];
    // the rows of a warp end together: num_centroids is a multiple of 32
    for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    m = fmaxf(m, s);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(reinterpret_cast<int*>(out + g), __float_as_int(m));
}

template <int D>
__global__ void __launch_bounds__(320, 1)
kmeans_assign_tc_kernel(const __grid_constant__ CUtensorMap tm_data, const __grid_constant__ CUtensorMap tm_cent,
                        const __grid_constant__ KmeansTcParams p) {
  using L = KmeansTcSmem<D>;
  constexpr uint32_t kTmemCols = 512;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work items: (group, 256 tokens), group by group so that the CTAs that run together share centroids in L2
  const int per_group = (p.num_tokens + kKtTokens - 1) / kKtTokens;
  const long long items = static_cast<long long>(p.groups) * per_group;
  auto mark_for_recheck = [&](long long from) {   // this CTA's items from `from` on go through the exact path
    for (long long it = from; it < items; it += gridDim.x) {
      const int g = static_cast<int>(it / per_group), t0 = static_cast<int>(it % per_group) * kKtTokens;
      for (int r = threadIdx.x; r < kKtTokens; r += blockDim.x)
        if (t0 + r < p.num_tokens) p.idx[static_cast<long long>(g) * p.num_tokens + t0 + r] = -1;
    }
    if (threadIdx.x == 0) atomicMax(p.flagged_count, p.flagged_cap + 1);   // forces the full sweep
  };
  if ((sbase & 1023u) || cta_device_failed()) {
    if ((sbase & 1023u) && threadIdx.x == 0) record_failure(400);
    mark_for_recheck(blockIdx.x);
    return;
  }
  const uint32_t a_s = sbase + L::kAOff, b_s = sbase + L::kBOff, bars = sbase + L::kBarOff;
  const uint32_t bar_a_full = bars, bar_a_empty = bars + 16, bar_b_full = bars + 32, bar_b_empty = bar_b_full + 8 * kKtStages;
  const uint32_t bar_s_full = bar_b_empty + 8 * kKtStages, bar_s_empty = bar_s_full + 32;
  volatile uint32_t* tmem_base_s = reinterpret_cast<volatile uint32_t*>(smem + L::kMiscOff);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  const int ntiles = (p.num_centroids + kKtCent - 1) / kKtCent;

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int i = 0; i < 2; ++i) { mbar_init(bar_a_full + 8 * i, 1); mbar_init(bar_a_empty + 8 * i, 8 + 1); }   // epilogue warps, tensor core
    for (int i = 0; i < 2 * kKtStages; ++i) mbar_init(bar_b_full + 8 * i, 1);
    for (int i = 0; i < 4; ++i) { mbar_init(bar_s_full + 8 * i, 1); mbar_init(bar_s_empty + 8 * i, 4); }
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_base_s)), kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s;

  // The barriers' phases run on over the items: `step` counts centroid tiles, `n` items.
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_data); tma_prefetch_desc(&tm_cent);
      bool ok = true;
      uint32_t step = 0, n = 0;
      for (long long it = blockIdx.x; ok && it < items; it += gridDim.x, ++n) {
        const int g = static_cast<int>(it / per_group), t0 = static_cast<int>(it % per_group) * kKtTokens;
        for (int j = 0; ok && j < ntiles; ++j, ++step) {
          const int st = step % kKtStages;
          if (step >= kKtStages) ok = mbar_wait(bar_b_empty + 8 * st, (step / kKtStages - 1) & 1, cta_abort, 401);
          if (!ok) break;
          mbar_expect_tx(bar_b_full + 8 * st, L::kBBytes);
#pragma unroll
          for (int h = 0; h < D / 64; ++h)
            tma_load_4d(b_s + st * L::kBBytes + h * (kKtCent * 128), &tm_cent, bar_b_full + 8 * st, h * 64, j * kKtCent, g, 0);
          if (j == 0) {
            const uint32_t ab = n & 1;   // an item's token tiles arrive while the one before it is worked on
            if (n >= 2) ok = mbar_wait(bar_a_empty + 8 * ab, ((n >> 1) - 1) & 1, cta_abort, 403);
            if (!ok) break;
            mbar_expect_tx(bar_a_full + 8 * ab, 2 * L::kABytes);
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
              for (int h = 0; h < D / 64; ++h)
                tma_load_4d(a_s + (2 * ab + a) * L::kABytes + h * (128 * 128), &tm_data, bar_a_full + 8 * ab, h * 64, t0 + a * 128, g, 0);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ tcgen05 issuer
    {  // converged warp, one elected lane issues (operands stay warp-uniform values)
      const uint32_t fmt = p.bf16 ? 1u : 0u;
      const uint32_t idesc = make_idesc(fmt, fmt, 0, 0, 128, kKtCent);
      bool ok = true;
      uint32_t step = 0, n = 0;
      for (long long it = blockIdx.x; ok && it < items; it += gridDim.x, ++n) {
        const uint32_t ab = n & 1;
        ok = mbar_wait_warp(bar_a_full + 8 * ab, (n >> 1) & 1, cta_abort, 411);
        for (int j = 0; ok && j < ntiles; ++j, ++step) {
          const int st = step % kKtStages, buf = step & 1;
          ok = mbar_wait_warp(bar_b_full + 8 * st, (step / kKtStages) & 1, cta_abort, 412);
          if (!ok) break;
          const uint64_t b_desc = smem_desc_sw128(b_s + st * L::kBBytes, 16, 1024);
          for (int a = 0; ok && a < 2; ++a) {
            if (step >= 2) ok = mbar_wait_warp(bar_s_empty + 16 * a + 8 * buf, ((step >> 1) - 1) & 1, cta_abort, 413);
            if (!ok) break;
            tc_fence_after();
            const uint64_t a_desc = smem_desc_sw128(a_s + (2 * ab + a) * L::kABytes, 16, 1024);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const uint32_t off_a = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
              const uint32_t off_b = (kk >> 2) * (kKtCent * 128) + (kk & 3) * 32;
              mma_ss_elect(tmem + (2 * a + buf) * kKtCent, a_desc + (off_a >> 4), b_desc + (off_b >> 4), idesc, kk > 0);
            }
            tc_commit_elect(bar_s_full + 16 * a + 8 * buf);
          }
          tc_commit_elect(bar_b_empty + 8 * st);
        }
        tc_commit_elect(bar_a_empty + 8 * ab);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: running top-2 per token
    const int a = (warp - 2) >> 2;              // token tile of this warp
    const int quarter = warp & 3;               // TMEM lanes this warp may touch: 32 * (warp % 4) ..
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    uint64_t column[16];                        // 32nds, for two scores at a time
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      column[c] = f32x2_pack(2 * c / 32.0f, (2 * c + 1) / 32.0f);
      asm volatile("" : "+l"(column[c]));       // in registers, not loaded for every use
    }
    const uint64_t whole = f32x2_pack(12582912.0f, 12582912.0f);
    bool ok = true;
    uint32_t step = 0, n = 0;
    for (long long it = blockIdx.x; it < items; it += gridDim.x, ++n) {
      const int g = static_cast<int>(it / per_group), tok = static_cast<int>(it % per_group) * kKtTokens + a * 128 + row;
      // |k|^2 of this thread's token, from the staged tile (16-byte chunk c of a row sits at c ^ (row & 7))
      const uint32_t ab = n & 1;
      ok = mbar_wait_warp(bar_a_full + 8 * ab, (n >> 1) & 1, cta_abort, 420);
      if (!ok) break;
      float nrm2 = 0.f;
      const uint8_t* arow = smem + L::kAOff + (2 * ab + a) * L::kABytes + row * 128;
#pragma unroll
      for (int ch = 0; ch < D / 8; ++ch) {
        const uint4 raw = *reinterpret_cast<const uint4*>(arow + (ch >> 3) * (128 * 128) + (((ch & 7) ^ (row & 7)) << 4));
        float f[8];
        if (p.bf16) unpack8<true>(raw, f); else unpack8<false>(raw, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) nrm2 += f[i] * f[i];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_a_empty + 8 * ab);
      const float scale = kKtScale / (sqrtf(nrm2) * sqrtf(p.max_cnorm2[g]));
      const uint64_t scale2 = f32x2_pack(scale, scale);
      float best = -INFINITY, second = -INFINITY;
      int best_chunk = 0;
      for (int j = 0; ok && j < ntiles; ++j, ++step) {
        const int buf = step & 1;
        ok = mbar_wait_warp(bar_s_full + 16 * a + 8 * buf, (step >> 1) & 1, cta_abort, 421);
        if (!ok) break;
        tc_fence_after();
        const uint32_t s_tmem = tmem + lane_addr + (2 * a + buf) * kKtCent;
        // num_centroids is a multiple of 32: a 32-column chunk is whole or absent
        const int nch = min(kKtCent / 32, (p.num_centroids - j * kKtCent) / 32);
        // The column rides in the score's 32nds, so the running maximum carries it along.  Two at a time: the larger against
        // the best, the rest against the second.
        auto scan = [&](const uint32_t (&r)[32], int chunk) {
          const float before = best;
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float v0, v1;
            const uint64_t u = f32x2_fma(f32x2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), scale2, whole);
            f32x2_unpack(f32x2_add(f32x2_sub(u, whole), column[c / 2]), v0, v1);
            const float hi = fmaxf(v0, v1), lo = fminf(v0, v1);
            second = max3(second, lo, fminf(best, hi));
            best = fmaxf(best, hi);
          }
          if (best > before) best_chunk = chunk;
        };
        // two register buffers: the load of the next chunk is in flight while this one is scanned
        uint32_t r0[32], r1[32];
        const int chunk0 = j * (kKtCent / 32);
        tmem_ld32(s_tmem, r0);
        if (nch == kKtCent / 32) {
#pragma unroll
          for (int ch = 0; ch < kKtCent / 32; ch += 2) {
            tmem_wait_ld();
            tmem_ld32(s_tmem + (ch + 1) * 32, r1);
            scan(r0, chunk0 + ch);
            tmem_wait_ld();
            if (ch + 2 < kKtCent / 32) tmem_ld32(s_tmem + (ch + 2) * 32, r0);
            scan(r1, chunk0 + ch + 1);
          }
        } else {
#pragma unroll 1
          for (int ch = 0; ch < nch; ++ch) {
            tmem_wait_ld();
            scan(r0, chunk0 + ch);
            if (ch + 1 < nch) tmem_ld32(s_tmem + (ch + 1) * 32, r0);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_s_empty + 16 * a + 8 * buf);
      }
      if (!ok) break;
      if (tok < p.num_tokens) {
        const long long at = static_cast<long long>(g) * p.num_tokens + tok;
        const int best_idx = best_chunk * 32 + (static_cast<int>(best * 32.0f) & 31);
        const bool sure = (best - second) > kKtGap && fminf(nrm2, p.max_cnorm2[g]) >= kKtMinNorm2;
        p.idx[at] = sure ? best_idx : (-1 - best_idx);
        if (!sure) {
          const int slot = atomicAdd(p.flagged_count, 1);
          if (slot < p.flagged_cap) p.flagged[slot] = static_cast<int>(at);
        }
      }
    }
  }

  // ------------------------------------------------------------------ tear-down (also after a wait gave up)
  if (*cta_abort) {
    const uint64_t t_wait = globaltimer_ns();
    while (globaltimer_ns() - t_wait < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (*cta_abort) mark_for_recheck(blockIdx.x);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// Exact re-scoring of the listed tokens, per_sweep consecutive ones of the list per CTA (the CTAs loop over the list).  A sweep
// serves those of one group; neighbours in a long list mostly belong to one, in a short one to several (the rule is at the launch):
//   1. fp32 scores of ALL centroids of the group into shared memory: mma.sync m16n8k16 with 16 centroid rows as A, straight
//      from global memory (16 bytes of a row per lane; the order of the channels inside a product does not matter), and the
//      tokens as the columns of B.  A token's own sweep with fp32 FMAs took 15 instructions per row for unpacking and shuffles
//      and one read of all centroids per token: 42-86 us for the tokens of an iteration (8 x 65536 keys, 1024 centroids), 30-32 us
//      like this, the latency of a sweep and of the fp64 chain; 4 x 262144 keys, 4096 centroids 400-950 and 153-302, 2 x 1048576,
//      16384 (two tokens a sweep) 4760-17800 and 3280-11770;
//   2. a warp per token: the candidates, i.e. centroids whose fp32 score lies within the error band of the largest one (the
//      same bound as in the assignment kernel, which also covers this pass's own rounding); a score that is not a number counts;
//   3. the candidates' exact scores in fp64 (exact products, index-order sum), the largest wins, the lowest index
//      on ties.  More than kMaxCand candidates (degenerate data, e.g. an all-zero key) take the fp64 path for every
//      centroid.
// When the list overflowed, every token whose idx is still negative is re-scored instead (a sweep over all
// tokens, the list is ignored).
constexpr int kRecheckTokens = 8;
constexpr int kMaxCand = 64;

template <int D, bool BF16>
__device__ __forceinline__ double exact_score(const double* kd, const uint8_t* row) {
  const uint4* x = reinterpret_cast<const uint4*>(row);
  double s = 0.0;
#pragma unroll 4
  for (int ch = 0; ch < D / 8; ++ch) {
    float f[8];
    unpack8<BF16>(x[ch], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += kd[ch * 8 + i] * static_cast<double>(f[i]);
  }
  return s;
}

// per_sweep <= kRecheckTokens, at most as many tokens as the scores' shared memory holds
template <int D, bool BF16>
__global__ void __launch_bounds__(256)
kmeans_recheck_list_kernel(const uint8_t* data, const uint8_t* cent, int* idx, const int* flagged, const int* flagged_count,
                           int flagged_cap, const float* max_cnorm2, int groups, int num_tokens, int num_centroids, int per_sweep) {
  extern __shared__ float score_s[];      // [per_sweep][num_centroids]
  __shared__ double kd_s[kRecheckTokens][D];
  __shared__ int cand_s[kRecheckTokens][kMaxCand];
  __shared__ int token_s[kRecheckTokens];  // g * num_tokens + t, -1: none
  static_assert(kRecheckTokens == 8, "a warp per token, a column of the matrix product per token");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = *flagged_count;
  const bool sweep = count > flagged_cap;
  const long long total = sweep ? static_cast<long long>(groups) * num_tokens : count;
  for (long long e0 = static_cast<long long>(blockIdx.x) * per_sweep; e0 < total; e0 += static_cast<long long>(gridDim.x) * per_sweep) {
    __syncthreads();
    if (threadIdx.x < kRecheckTokens) {
      const long long e = e0 + threadIdx.x;
      int at = -1;
      if (threadIdx.x < per_sweep && e < total) {
        at = sweep ? static_cast<int>(e) : flagged[e];
        if (sweep && idx[at] >= 0) at = -1;
      }
      token_s[threadIdx.x] = at;
    }
    __syncthreads();
    unsigned left = 0;
#pragma unroll
    for (int j = 0; j < kRecheckTokens; ++j) left |= token_s[j] >= 0 ? 1u << j : 0u;
    while (left) {
      // the tokens of the first one's group
      const int g = token_s[__ffs(left) - 1] / num_tokens;
      unsigned mine = 0;
#pragma unroll
      for (int j = 0; j < kRecheckTokens; ++j) mine |= (left >> j & 1u) && token_s[j] / num_tokens == g ? 1u << j : 0u;
      left &= ~mine;
      const uint8_t* cg = cent + static_cast<long long>(g) * num_centroids * D * 2;
      // 1. lane (r, c) = (lane / 4, lane % 4) reads channels 8 (4 q + c) .. + 7: of token r for B, of rows r and r + 8 for A
      const int r = lane >> 2, c = lane & 3;
      uint4 b[D / 32];
#pragma unroll
      for (int q = 0; q < D / 32; ++q)
        b[q] = mine >> r & 1u ? *reinterpret_cast<const uint4*>(data + (static_cast<long long>(token_s[r]) * D + 8 * (4 * q + c)) * 2)
                              : make_uint4(0, 0, 0, 0);
      for (int row0 = warp * 16; row0 < num_centroids; row0 += 8 * 16) {
        uint4 a0[D / 32], a1[D / 32];
        const uint8_t* row = cg + (static_cast<long long>(row0 + r) * D + 8 * c) * 2;
#pragma unroll
        for (int q = 0; q < D / 32; ++q) {
          a0[q] = *reinterpret_cast<const uint4*>(row + q * 64);
          a1[q] = *reinterpret_cast<const uint4*>(row + q * 64 + 8 * D * 2);
        }
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < D / 32; ++q) {
          const uint32_t lo[4] = {a0[q].x, a1[q].x, a0[q].y, a1[q].y}, hi[4] = {a0[q].z, a1[q].z, a0[q].w, a1[q].w};
          mma_16816<BF16>(s, lo, b[q].x, b[q].y);
          mma_16816<BF16>(s, hi, b[q].z, b[q].w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)   // rows r, r, r + 8, r + 8 of tokens 2 c, 2 c + 1
          if (mine >> (2 * c + (i & 1)) & 1u) score_s[(2 * c + (i & 1)) * num_centroids + row0 + r + 8 * (i >> 1)] = s[i];
      }
      // the token as fp64, and its norm
      float nrm2 = 0.f;
      if (mine >> warp & 1u) {
        const uint8_t* krow = data + static_cast<long long>(token_s[warp]) * D * 2;
        for (int ch = lane; ch < D; ch += 32) {
          const float f = to_f32<BF16>(reinterpret_cast<const uint16_t*>(krow)[ch]);
          kd_s[warp][ch] = static_cast<double>(f);
          nrm2 += f * f;
        }
        for (int o = 16; o > 0; o >>= 1) nrm2 += __shfl_xor_sync(0xffffffffu, nrm2, o);
      }
      __syncthreads();
      if (mine >> warp & 1u) {
        const float* score = score_s + warp * num_centroids;
        const double* kd = kd_s[warp];
        // 2. candidates inside the error band; without a band (norms beyond fp32 squares either way) none is left out
        float mx = -INFINITY;
        for (int k = lane; k < num_centroids; k += 32) mx = fmaxf(mx, score[k]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float cnorm2 = max_cnorm2[g];
        const float tol = fminf(nrm2, cnorm2) >= kKtMinNorm2 ? kKtTol * sqrtf(nrm2) * sqrtf(cnorm2) : INFINITY;
        int ncand = 0;
        for (int k = lane; k < num_centroids; k += 32) {   // num_centroids is a multiple of 32
          const bool near = !(score[k] < mx - tol);
          const unsigned votes = __ballot_sync(0xffffffffu, near);
          const int slot = ncand + __popc(votes & ((1u << lane) - 1u));
          if (near && slot < kMaxCand) cand_s[warp][slot] = k;
          ncand += __popc(votes);
        }
        __syncwarp();
        // 3. exact scores; a lane's centroids ascend, so the lowest index is kept on ties
        double best = -1.0 / 0.0;
        int bi = 0x7fffffff;
        const bool listed = ncand <= kMaxCand;
        for (int k = lane; k < (listed ? ncand : num_centroids); k += 32) {
          const int cand = listed ? cand_s[warp][k] : k;
          const double sc = exact_score<D, BF16>(kd, cg + static_cast<long long>(cand) * D * 2);
          if (sc > best || (sc == best && cand < bi)) { best = sc; bi = cand; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) idx[token_s[warp]] = bi < num_centroids ? bi : 0;   // no candidate at all: a NaN key
      }
      __syncthreads();
    }
  }
}

// ---- member sums that do not depend on the order of the members ------------------------------------------------
// counts[g, c] += members of cluster c and slot[g, t] = the arrival rank of token t inside its cluster.  The rank
// depends on timing, the sums below do not: adding 16-bit values in fp64 is exact in any order.  2048 tokens of a group are
// ranked in a CTA's shared memory, and a cluster that occurs among them takes one global atomic: clusters are uneven (the first
// iterations' centroids have very different norms, and one of them can attract a tenth of the tokens), and an address takes its
// atomics one after another.  8 x 65536 tokens, 1024 clusters: 3.8 us, 16.7 with an atomic per cluster and warp; 4 x 262144
// tokens, 8192 clusters: 10 and 19.  With more clusters a CTA's pass over its counters outweighs that (32768: 49 and 19 us).
constexpr int kCountTokens = 2048, kCountThreads = 512, kCountMaxClusters = 8192;
__global__ void __launch_bounds__(kCountThreads) kmeans_count_kernel(const int* idx, int* counts, int* slot, int num_tokens, int num_centroids) {
  extern __shared__ int cnt_s[];               // [num_centroids]
  constexpr int kPer = kCountTokens / kCountThreads;
  const int t0 = blockIdx.y * kCountTokens + threadIdx.x;
  const long long first = static_cast<long long>(blockIdx.x) * num_tokens;
  int* total = counts + static_cast<long long>(blockIdx.x) * num_centroids;
  int c[kPer], rank[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) c[u] = t0 + u * kCountThreads < num_tokens ? idx[first + t0 + u * kCountThreads] : -1;
  for (int k = threadIdx.x; k < num_centroids; k += kCountThreads) cnt_s[k] = 0;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPer; ++u) rank[u] = c[u] >= 0 ? atomicAdd(cnt_s + c[u], 1) : 0;
  __syncthreads();
  for (int k = threadIdx.x; k < num_centroids; k += kCountThreads)
    if (cnt_s[k] > 0) cnt_s[k] = atomicAdd(total + k, cnt_s[k]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPer; ++u)
    if (c[u] >= 0) slot[first + t0 + u * kCountThreads] = cnt_s[c[u]] + rank[u];
}
// The same for many clusters: the lanes of a warp that hold the same cluster share one global atomic.
__global__ void kmeans_count_many_kernel(const int* idx, int* counts, int* slot, long long total, int num_tokens, int num_centroids) {
  const int lane = threadIdx.x & 31;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i - lane < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const bool live = i < total;
    // (cluster of the group) as one number: groups * num_centroids is below 2^31 (the counts are an int array)
    const int key = live ? static_cast<int>(i / num_tokens) * num_centroids + idx[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(same) - 1, rank = __popc(same & ((1u << lane) - 1u));
    int base = 0;
    if (live && lane == leader) base = atomicAdd(counts + key, __popc(same));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (live) slot[i] = base + rank;
  }
}
// offsets[g, c] = exclusive prefix sum of counts[g, :]: one CTA per group
__global__ void __launch_bounds__(1024) kmeans_offsets_kernel(const int* counts, int* offsets, int num_centroids) {
  __shared__ int warp_tot[32];
  __shared__ int carry_s;
  const int g = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* cg = counts + static_cast<long long>(g) * num_centroids;
  int* og = offsets + static_cast<long long>(g) * num_centroids;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int base = 0; base < num_centroids; base += 1024) {
    const int c = base + threadIdx.x;
    const int v = c < num_centroids ? cg[c] : 0;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int before = carry_s;
    for (int w = 0; w < warp; ++w) before += warp_tot[w];
    if (c < num_centroids) og[c] = before + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = before + incl;
    __syncthreads();
  }
}
__global__ void kmeans_scatter_kernel(const int* idx, const int* slot, const int* offsets, int* members, long long total,
                                      int num_tokens, int num_centroids) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int g = static_cast<int>(i / num_tokens);
    const int c = idx[i];
    members[static_cast<long long>(g) * num_tokens + offsets[static_cast<long long>(g) * num_centroids + c] + slot[i]] =
        static_cast<int>(i - static_cast<long long>(g) * num_tokens);
  }
}
// sums[g, c, :] += x[g, t, :] over the members, in fp64 (the caller has zeroed sums).  HBM-bound: one read of x.  The
// unit of work is kSumRows consecutive entries of the group's member list, NOT a cluster: a warp per cluster left the
// chip waiting for the warp of the largest one (851 us on average at 8 x 65536 keys in 1024 clusters whose largest held
// thousands; 42 us now, and 21 us for reading the keys once from HBM).  A warp adds rows of one cluster in registers and hands
// the sum over when the cluster changes: a cluster that lies wholly inside the warp's range is stored, the first and
// the last one of a range may be shared with the neighbours and are added with fp64 atomics (exact, so the order of
// arrival does not matter).  All 32 lanes read one row (8 or 4 bytes each), eight rows in flight.
constexpr int kSumRows = 64;
template <int D, bool BF16>
__global__ void __launch_bounds__(256)
kmeans_member_sum_kernel(const uint8_t* x, const int* idx, const int* members, double* sums, int groups, int num_tokens,
                         int num_centroids) {
  constexpr int kPer = D / 32;                 // channels per lane
  constexpr int kInFlight = 8;
  const int chunks = (num_tokens + kSumRows - 1) / kSumRows;
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= static_cast<long long>(groups) * chunks) return;
  const int g = static_cast<int>(w / chunks), p0 = static_cast<int>(w % chunks) * kSumRows;
  const int n = min(kSumRows, num_tokens - p0);
  const int* mem = members + static_cast<long long>(g) * num_tokens + p0;
  const int* cl = idx + static_cast<long long>(g) * num_tokens;
  const uint8_t* xg = x + static_cast<long long>(g) * num_tokens * D * 2 + lane * kPer * 2;
  double* out = sums + static_cast<long long>(g) * num_centroids * D + lane * kPer;
  int tok[kSumRows / 32], clu[kSumRows / 32];
#pragma unroll
  for (int u = 0; u < kSumRows / 32; ++u) {
    const bool live = lane + 32 * u < n;
    tok[u] = live ? mem[lane + 32 * u] : 0;
    clu[u] = live ? cl[tok[u]] : -1;
  }
  const double scale = narrow_scale<BF16>();
  double acc[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) acc[i] = 0.0;
  int cur = __shfl_sync(0xffffffffu, clu[0], 0);
  bool first = true;
#pragma unroll
  for (int u = 0; u < kSumRows / 32; ++u) {
#pragma unroll 1
    for (int r0 = 0; r0 < 32; r0 += kInFlight) {
      if (u * 32 + r0 >= n) break;
      uint32_t v[kInFlight][kPer / 2];
#pragma unroll
      for (int q = 0; q < kInFlight; ++q) {
        // rows past the end read row 0 of the group; their cluster is -1 and they are not added
        const long long off = static_cast<long long>(__shfl_sync(0xffffffffu, tok[u], r0 + q)) * D * 2;
        if (kPer == 4) {
          const uint2 t = *reinterpret_cast<const uint2*>(xg + off);
          v[q][0] = t.x; v[q][kPer / 2 - 1] = t.y;
        } else {
          v[q][0] = *reinterpret_cast<const uint32_t*>(xg + off);
        }
      }
#pragma unroll
      for (int q = 0; q < kInFlight; ++q) {
        const int c = __shfl_sync(0xffffffffu, clu[u], r0 + q);
        if (c < 0) continue;
        if (c != cur) {
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            if (first) atomicAdd(out + static_cast<long long>(cur) * D + i, acc[i]);
            else out[static_cast<long long>(cur) * D + i] = acc[i];
            acc[i] = 0.0;
          }
          first = false;
          cur = c;
        }
        bool special = false;                  // infinities and NaNs have no exponent of their own in the shifted form
#pragma unroll
        for (int i = 0; i < kPer / 2; ++i) special |= narrow_special<BF16>(v[q][i]);
        if (!special) {
#pragma unroll
          for (int i = 0; i < kPer / 2; ++i) {
            acc[2 * i] = fma(narrow_as_double<BF16>(v[q][i] & 0xffffu), scale, acc[2 * i]);
            acc[2 * i + 1] = fma(narrow_as_double<BF16>(v[q][i] >> 16), scale, acc[2 * i + 1]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < kPer / 2; ++i) {
            acc[2 * i] += static_cast<double>(to_f32<BF16>(static_cast<uint16_t>(v[q][i] & 0xffffu)));
            acc[2 * i + 1] += static_cast<double>(to_f32<BF16>(static_cast<uint16_t>(v[q][i] >> 16)));
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) atomicAdd(out + static_cast<long long>(cur) * D + i, acc[i]);
}

// ---- member lists in token order: a stable counting sort -------------------------------------------------------
// (triton_reverse_index, kmeans.py:199-262, whose own order is the atomic arrival order.)  A group's tokens are cut into
// at most kSortRanges ranges; one warp per (range, group) walks its range in token order.  Pass 1 counts the clusters of
// every range, a scan over the ranges turns the counts into first positions, pass 2 walks again and writes
// clusters[g, c, position].  Linear in the tokens, where ranking the members of a cluster against each other is
// quadratic in the cluster's size (8 x 65536 tokens, 1024 clusters: 25 us for the three, 90 us for count, scatter and
// ranking before).
// The counters of the clusters [c0, c0 + nc) live in shared memory (nc ints); more than kSortClusters go in several calls.
constexpr int kSortRanges = 64;
constexpr int kSortClusters = 49152;

// hist[g, r, c] = members of cluster c among the tokens of range r
__global__ void __launch_bounds__(32) kmeans_range_count_kernel(const int* idx, int* hist, int num_tokens, int num_centroids, int per_range,
                                                                int c0, int nc) {
  extern __shared__ int cnt_s[];
  const int g = blockIdx.x, r = blockIdx.y, lane = threadIdx.x;
  for (int c = lane; c < nc; c += 32) cnt_s[c] = 0;
  __syncwarp();
  const int t0 = r * per_range, t1 = min(num_tokens, t0 + per_range);
  const int* ig = idx + static_cast<long long>(g) * num_tokens;
#pragma unroll 4
  for (int t = t0 + lane; t < t1; t += 32) {
    const int c = ig[t] - c0;
    if (c >= 0 && c < nc) atomicAdd(cnt_s + c, 1);
  }
  __syncwarp();
  int* hg = hist + (static_cast<long long>(g) * gridDim.y + r) * num_centroids + c0;
  for (int c = lane; c < nc; c += 32) hg[c] = cnt_s[c];
}
// hist[g, r, c] <- members of c in the ranges before r;  cluster_size[g, c] = all of them.  A thread per cluster.
__global__ void __launch_bounds__(256) kmeans_range_scan_kernel(int* hist, int* cluster_size, int ranges, int num_centroids) {
  const int c = blockIdx.y * 256 + threadIdx.x, g = blockIdx.x;
  if (c >= num_centroids) return;
  int* h = hist + static_cast<long long>(g) * ranges * num_centroids + c;
  int run = 0;
  for (int r0 = 0; r0 < ranges; r0 += 8) {
    int v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = r0 + u < ranges ? h[static_cast<long long>(r0 + u) * num_centroids] : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (r0 + u < ranges) { h[static_cast<long long>(r0 + u) * num_centroids] = run; run += v[u]; }
  }
  cluster_size[static_cast<long long>(g) * num_centroids + c] = run;
}
// Pass 2.  A warp takes 32 tokens at a time: a token's position is its cluster's next free one plus the number of lower
// lanes that hold the same cluster.
__global__ void __launch_bounds__(32) kmeans_range_emit_kernel(const int* idx, const int* hist, int* clusters, int num_tokens,
                                                               int num_centroids, int per_range, int max_cluster_size,
                                                               int c0, int nc) {
  extern __shared__ int next_s[];
  const int g = blockIdx.x, r = blockIdx.y, lane = threadIdx.x;
  const int* hg = hist + (static_cast<long long>(g) * gridDim.y + r) * num_centroids + c0;
  for (int c = lane; c < nc; c += 32) next_s[c] = hg[c];
  __syncwarp();
  const int t0 = r * per_range, t1 = min(num_tokens, t0 + per_range);
  const int* ig = idx + static_cast<long long>(g) * num_tokens;
  int* out = clusters + (static_cast<long long>(g) * num_centroids + c0) * max_cluster_size;
  int ahead = t0 + lane < t1 ? ig[t0 + lane] : -1;
  for (int base = t0; base < t1; base += 32) {
    const int c = (ahead >= c0 && ahead - c0 < nc) ? ahead - c0 : -1;
    ahead = base + 32 + lane < t1 ? ig[base + 32 + lane] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (c >= 0) {
      const int pos = next_s[c] + rank;
      if (pos < max_cluster_size) out[static_cast<long long>(c) * max_cluster_size + pos] = base + lane;
    }
    __syncwarp();
    if (c >= 0 && rank == 0) next_s[c] += __popc(same);
    __syncwarp();
  }
}

}  // namespace sq
