// Relative-distance attention-energy histogram (window_search.cuh states the rule) on the 5th-generation tensor cores,
// in ONE sweep over the keys of a row block.
//
// What bounds it: one exponential per (query, key) pair.  The mma.sync kernel swept the keys twice (statistics, then
// normalised weights), computed two exponentials and an IEEE division per pair and took 10.6 ms for 28 heads x 8192
// tokens x 200 bins (this one 1.11 ms); the products of one sweep are 0.15 ms of the measured tensor rate, its exponentials 0.2 ms of the
// special-function units.  Hence:
//   * a thread owns one query row (a TMEM lane) and meets its keys in order, so its bins never increase: a bin is one
//     run, kept as A0 = sum a and A1 = sum a * (ref - j) with a = 2^(score - base) NOT normalised, and stored once, in a
//     per-row histogram in shared memory; the row sum is known at the end and scales the stored bins then.  ref is the last
//     visible key met so far: the run's weighted sum A0 * w(ref) + A1 * (bins per key) has no negative term, so nothing
//     cancels however narrow the bins are (relative to the first key of a chunk, rows of 8 keys with 200 bins were off by
//     4e-6, 3e-7 so).  base is the maximum of the row's first keys; fp32 holds a up to 2^60 above it, so it moves (and the
//     stored bins are rescaled) only past that.
//   * the bin of a key is not computed per pair: the run knows the first key of the next bin, from integer arithmetic
//     that steps from one bin's edge to the next, and from how the reference's fp32 expression rounds where an edge is a
//     whole number of keys (edge()).
//   * one CTA = 128 rows of one head.  The keys up to the diagonal are cut in four parts at 64-key tiles: four epilogue
//     warps walk each, with two 64-column accumulators, so that sixteen warps hide the latencies of a row's chain although
//     the per-row histogram (nbins x 128 fp32) leaves room for one CTA (two parts, eight warps: 1.70 ms).
//     A bin in which parts meet is the only one that several write; a part keeps its first run aside.
//   warp 0 TMA producer, warp 1 tcgen05 issuer (owns the 512 TMEM columns).
#pragma once
#include <cuda.h>

#include "ptx.cuh"
#include "window_search.cuh"

namespace sq {

constexpr int kWtRows = 128, kWtKeys = 64, kWtParts = 4;
constexpr int kWtThreads = 64 + kWtParts * 128;
constexpr int kWtMaxBins = 248;       // nbins x 128 fp32 + Q tile + one K stage per part within 227 KB
constexpr int kWtKeysPerBin = 1024;   // seq_len / nbins at most this (edge(): at most one distance near an edge)
constexpr float kWtLazyLog2 = 60.0f;

template <int D>
struct WindowTcSmem {
  static constexpr int kQBytes = kWtRows * D * 2;
  static constexpr int kTileBytes = kWtKeys * D * 2;
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kQBytes;                                    // one stage per part
  static constexpr int kFacOff = kKOff + kWtParts * kTileBytes;            // [parts][128] fp32: base, sum, factor
  static constexpr int kFirstOff = kFacOff + kWtParts * 128 * 4;           // [parts][128] int: first bin
  static constexpr int kAsideOff = kFirstOff + kWtParts * 128 * 4;         // [parts][128] fp32: its value
  static constexpr int kTieOff = kAsideOff + kWtParts * 128 * 4;           // [256] bytes
  static constexpr int kBarOff = kTieOff + 256;                            // q_full, k_full[parts], s_full[parts][2], s_empty[parts][2]
  static constexpr int kBars = 1 + 5 * kWtParts;
  static constexpr int kMiscOff = kBarOff + 8 * kBars;
  static constexpr int kHistOff = (kMiscOff + 8 + 15) / 16 * 16;           // 16-byte aligned; [nbins][128]
  static size_t total(int nbins) { return kHistOff + static_cast<size_t>(nbins) * 128 * sizeof(float); }
  static_assert(kHistOff % 16 == 0, "the histogram is cleared with 16-byte stores");
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// One query row's walk over its keys.
struct WindowRow {
  int i, sink, nbins;
  float ctx, cinv;           // max(i - sink, 1), bins per key (0 for rows without bins of their own)
  float c2;                  // scores are raw dot products: exp(s * scale) = 2^(s * c2)
  float* hist;               // this row's column of [nbins][128]
  float* aside;              // where a later part's first run goes (the part before may write the same bin); first part: null
  float* slot;               // where the current run goes when it ends: its bin of `hist`, or aside
  const uint8_t* tie;        // [nbins] see edge()
  float base;                // raw score that the weights are relative to; -inf: no key yet
  float a0, a1, l;           // the current run (a1 relative to the current chunk's last visible key), sum of the finished runs
  int cur, next, first;      // bin of the current run (-1: none yet), first key behind it, bin of the first run
  int eq, er;                // the current bin's lower edge, cur * ctx = eq * nbins + er keys away
  int dq, dr;                // ctx = dq * nbins + dr: one bin
  int near_tie;              // edges this close (in er) to a whole number of keys need the reference's expression

  __device__ __forceinline__ int exact_bin(int dist) const {   // the reference's fp32 expressions (window_search.py:262-272)
    const float rel = (i <= sink) ? 0.f : __fdiv_rn(static_cast<float>(dist), ctx);
    return min(max(static_cast<int>(floorf(__fmul_rn(rel, static_cast<float>(nbins)))), 0), nbins - 1);
  }
  // First key whose bin is below cur, i.e. behind the smallest distance d with exact_bin(d) >= cur.  In real numbers that
  // is ceil(cur * ctx / nbins).  The reference's expression is within 3e-5 bins of the true quotient, so it can disagree
  // only at a distance whose quotient is that close to cur: with less than 32768 keys in the row only where the edge is a
  // whole number of keys, and there the quotient is cur / nbins in every row, so a table per bin says how it rounds.
  __device__ __forceinline__ void edge() {
    if (cur <= 0) { next = 0x7fffffff; return; }
    next = i - eq;
    if (near_tie == 0) {
      if (er == 0) next += tie[cur];
    } else if (er <= near_tie) {
      if (exact_bin(eq) >= cur) ++next;
    } else if (nbins - er <= near_tie) {
      if (exact_bin(eq + 1) < cur) --next;
    }
  }
  __device__ __forceinline__ void start(int dist) {
    cur = exact_bin(dist);
    eq = cur * static_cast<int>(ctx);                 // <= 2^18 * 2^8
    er = eq % nbins; eq /= nbins;
    edge();
  }
  __device__ __forceinline__ void begin(int j) {      // the first run behind the sink
    start(i - j);
    first = cur;
    slot = aside ? aside : hist + cur * 128;
  }
  __device__ __forceinline__ void lower() {           // one bin down
    --cur;
    eq -= dq; er -= dr;
    if (er < 0) { er += nbins; --eq; }
    slot = hist + cur * 128;
    edge();
  }
  __device__ __forceinline__ void flush(float t0) {   // t0 = weight at the key that a1 is relative to
    *slot = __fmaf_rn(a0, t0, cinv * a1);
    l += a0;
  }
  __device__ __forceinline__ float weight(int j) const { return __fmaf_rn(static_cast<float>(i - j), cinv, 1.0f); }
  __device__ __forceinline__ void look_at_max(float mx) {
    if (mx > base && (base == -INFINITY || (mx - base) * c2 > kWtLazyLog2)) {
      if (base != -INFINITY) {
        const float f = ex2_approx((base - mx) * c2);
        a0 *= f; a1 *= f; l *= f;
        if (cur >= 0)
          for (int b = cur + 1; b < (aside ? first : nbins); ++b) hist[b * 128] *= f;
        if (aside) *aside *= f;
      }
      base = mx;
    }
  }
  __device__ __forceinline__ float shift() const { return base == -INFINITY ? 0.f : -(base * c2); }

  // 32 keys from c0 on, all of them visible and behind the sink, bins wider than kSub keys: at most one edge among kSub
  // consecutive keys.  The lanes' edges lie all over the chunk, so every group of kSub keys splits its sums at the edge by
  // predicate, and the lanes that have one there end their runs together.
  template <int kSub>
  __device__ __forceinline__ void chunk32(const uint32_t (&r)[32], int c0) {
    float mx = max3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
#pragma unroll
    for (int c = 3; c < 31; c += 2) mx = max3(mx, __uint_as_float(r[c]), __uint_as_float(r[c + 1]));
    look_at_max(fmaxf(mx, __uint_as_float(r[31])));
    if (cur < 0) begin(c0);
    const float sh = shift(), t0 = weight(c0 + 31);
    a1 = __fmaf_rn(32.0f, a0, a1);
    float x[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) x[c] = ex2_approx(__fmaf_rn(__uint_as_float(r[c]), c2, sh));
#pragma unroll
    for (int s = 0; s < 32; s += kSub) {
      const int nb = next - c0;
      float v0 = 0.f, v1 = 0.f;
#pragma unroll
      for (int c = s; c < s + kSub; ++c) {
        if (c < nb) { a0 += x[c]; a1 = __fmaf_rn(x[c], static_cast<float>(31 - c), a1); }
        else { v0 += x[c]; v1 = __fmaf_rn(x[c], static_cast<float>(31 - c), v1); }
      }
      if (nb < s + kSub) {
        flush(t0);
        a0 = v0; a1 = v1;
        lower();
      }
    }
  }
  // 8 keys from c0 on, any of them past the row or in the sink, bins of any width
  __device__ __forceinline__ void chunk8(const uint32_t (&r)[8], int c0) {
    if (c0 > i) return;
    float mx = __uint_as_float(r[0]);
#pragma unroll
    for (int e = 1; e < 8; ++e) mx = (c0 + e <= i) ? fmaxf(mx, __uint_as_float(r[e])) : mx;
    look_at_max(mx);
    const int last = min(7, i - c0);
    const float sh = shift(), t0 = weight(c0 + last), to_last = static_cast<float>(last);
    a1 = __fmaf_rn(to_last + 1.0f, a0, a1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = c0 + e;
      const float x = ex2_approx(__fmaf_rn(__uint_as_float(r[e]), c2, sh));
      if (j < sink) {
        if (j <= i) l += x;
      } else if (j <= i) {
        if (j >= next) {
          flush(t0);
          a0 = a1 = 0.f;
          if (dq >= 1) {              // bins of a key or more: a rounded edge can leave one empty, hardly ever
            lower();
            while (j >= next) lower();
          } else {
            start(i - j);
            slot = hist + cur * 128;
          }
        } else if (cur < 0) {
          begin(j);
        }
        a0 += x;
        a1 = __fmaf_rn(x, to_last - static_cast<float>(e), a1);
      }
    }
  }
};

template <int D>
__global__ void __launch_bounds__(kWtThreads, 1)
window_hist_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ WindowHistParams p, int bf16) {
  using L = WindowTcSmem<D>;
  constexpr uint32_t kTmemCols = 512;   // accumulator u of part g: columns (2 g + u) * 64
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heads fastest: the heads of a KV group share K tiles in L2; the longest row blocks go first
  const int nblk = (p.n + kWtRows - 1) / kWtRows;
  const int blk = nblk - 1 - static_cast<int>(blockIdx.x) / p.hq, head = static_cast<int>(blockIdx.x) % p.hq;
  const int kvh = head / p.groups, i0 = blk * kWtRows;
  double* out = p.hist + static_cast<long long>(head) * p.nbins;
  auto poison = [&]() {   // this CTA cannot deliver its rows
    for (int b = threadIdx.x; b < p.nbins; b += blockDim.x) atomicAdd(out + b, __longlong_as_double(0x7ff8000000000000ll));
  };
  if ((sbase & 1023u) || cta_device_failed()) {
    if ((sbase & 1023u) && threadIdx.x == 0) record_failure(500);
    poison();
    return;
  }
  const uint32_t q_s = sbase + L::kQOff, k_s = sbase + L::kKOff, bars = sbase + L::kBarOff;
  const uint32_t bar_q = bars, bar_k = bars + 8, bar_s_full = bar_k + 8 * kWtParts, bar_s_empty = bar_s_full + 16 * kWtParts;   // [g], [2 g + u]
  volatile uint32_t* tmem_base_s = reinterpret_cast<volatile uint32_t*>(smem + L::kMiscOff);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  float* fac_s = reinterpret_cast<float*>(smem + L::kFacOff);
  int* first_s = reinterpret_cast<int*>(smem + L::kFirstOff);
  float* aside_s = reinterpret_cast<float*>(smem + L::kAsideOff);
  uint8_t* tie_s = smem + L::kTieOff;
  float* hist = reinterpret_cast<float*>(smem + L::kHistOff);
  const int ntiles = (min(i0 + kWtRows, p.n) + kWtKeys - 1) / kWtKeys;     // key tiles up to the diagonal
  auto part_begin = [&](int g) { return ntiles * g / kWtParts; };
  const int longest = (ntiles + kWtParts - 1) / kWtParts;

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int b = 0; b < 1 + 3 * kWtParts; ++b) mbar_init(bars + 8 * b, 1);
    for (int b = 1 + 3 * kWtParts; b < L::kBars; ++b) mbar_init(bars + 8 * b, 128);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_base_s)), kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  if (threadIdx.x < kWtParts * 128) aside_s[threadIdx.x] = 0.f;
  for (int b = threadIdx.x; b < p.nbins; b += kWtThreads)   // how the reference's expression rounds an edge that is a whole number of keys
    tie_s[b] = floorf(__fmul_rn(__fdiv_rn(static_cast<float>(b), static_cast<float>(p.nbins)), static_cast<float>(p.nbins))) >= b ? 1 : 0;
  for (int c = threadIdx.x; c < p.nbins * 32; c += kWtThreads) reinterpret_cast<uint4*>(hist)[c] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s;

  float row_l = 0.f, row_base = -INFINITY;   // of an epilogue thread's part of its row, for the combination below

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k);
      mbar_expect_tx(bar_q, L::kQBytes);
#pragma unroll
      for (int h = 0; h < D / 64; ++h) tma_load_4d(q_s + h * (kWtRows * 128), &tm_q, bar_q, h * 64, i0, head, 0);
      bool ok = true;
      for (int u = 0; ok && u < longest; ++u)
        for (int g = 0; ok && g < kWtParts; ++g) {
          const int tile = part_begin(g) + u;
          if (tile >= part_begin(g + 1)) continue;
          // the part's stage was last read by the products of its tile u - 1
          if (u >= 1) ok = mbar_wait(bar_s_full + 8 * (2 * g + ((u - 1) & 1)), ((u - 1) >> 1) & 1, cta_abort, 501);
          if (!ok) break;
          mbar_expect_tx(bar_k + 8 * g, L::kTileBytes);
#pragma unroll
          for (int h = 0; h < D / 64; ++h)
            tma_load_4d(k_s + g * L::kTileBytes + h * (kWtKeys * 128), &tm_k, bar_k + 8 * g, h * 64, tile * kWtKeys, kvh, 0);
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ tcgen05 issuer (converged warp, one elected lane)
    const uint32_t fmt = bf16 ? 1u : 0u;
    const uint32_t idesc = make_idesc(fmt, fmt, 0, 0, kWtRows, kWtKeys);
    const uint64_t q_desc = smem_desc_sw128(q_s, 16, 1024);
    bool ok = mbar_wait_warp(bar_q, 0, cta_abort, 511);
    for (int u = 0; ok && u < longest; ++u)
      for (int g = 0; ok && g < kWtParts; ++g) {
        if (part_begin(g) + u >= part_begin(g + 1)) continue;
        ok = mbar_wait_warp(bar_k + 8 * g, u & 1, cta_abort, 512);
        if (ok && u >= 2) ok = mbar_wait_warp(bar_s_empty + 8 * (2 * g + (u & 1)), ((u - 2) >> 1) & 1, cta_abort, 513);
        if (!ok) break;
        tc_fence_after();
        const uint64_t k_desc = smem_desc_sw128(k_s + g * L::kTileBytes, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off_q = ((kk >> 2) * (kWtRows * 128) + (kk & 3) * 32) >> 4, off_k = ((kk >> 2) * (kWtKeys * 128) + (kk & 3) * 32) >> 4;
          mma_ss_elect(tmem + (2 * g + (u & 1)) * kWtKeys, q_desc + off_q, k_desc + off_k, idesc, kk > 0);
        }
        tc_commit_elect(bar_s_full + 8 * (2 * g + (u & 1)));
      }
  } else {
    // ------------------------------------------------------------------ epilogue: one row per thread, part g of its keys
    const int g = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int i_first = i0 + quarter * 32;                              // the warp's first row
    WindowRow w;
    w.i = i0 + row < p.n ? i0 + row : -1;                               // rows past the end see no key
    w.sink = p.sink; w.nbins = p.nbins;
    const int ctx = max(w.i - p.sink, 1);
    w.ctx = static_cast<float>(ctx);
    w.cinv = w.i <= p.sink ? 0.f : __fdiv_rn(static_cast<float>(p.nbins), w.ctx);
    w.dq = ctx / p.nbins; w.dr = ctx % p.nbins;
    w.near_tie = static_cast<int>(3.2e-5f * w.ctx);
    w.c2 = p.scale * 1.44269504f;
    w.hist = hist + row; w.aside = g ? aside_s + g * 128 + row : nullptr; w.slot = w.hist; w.tie = tie_s;
    w.base = -INFINITY; w.a0 = w.a1 = w.l = 0.f; w.cur = w.first = -1; w.next = 0x7fffffff;
    w.eq = w.er = 0;
    // bins of 9 (17) keys and more: their edges are at least 8 (16) keys apart, rounded or not
    const bool wide = i_first + 31 < p.n && i_first - p.sink >= 9 * p.nbins, very_wide = wide && i_first - p.sink >= 17 * p.nbins;
    bool ok = true;
    int ref = 0;                                                        // first key not met yet
    const int tile0 = part_begin(g), tiles = part_begin(g + 1) - tile0;
    for (int u = 0; u < tiles; ++u) {
      const uint32_t slot = 2 * g + (u & 1);
      ok = mbar_wait_warp(bar_s_full + 8 * slot, (u >> 1) & 1, cta_abort, 521);
      if (!ok) break;
      tc_fence_after();
      const uint32_t s_tmem = tmem + lane_addr + slot * kWtKeys;
      const int j0 = (tile0 + u) * kWtKeys;
#pragma unroll 1
      for (int c = 0; c < kWtKeys;) {
        if (wide && (c & 31) == 0 && j0 + c >= p.sink && j0 + c + 31 <= i_first) {
          uint32_t r[32];
          tmem_ld32(s_tmem + c, r);
          tmem_wait_ld();
          if (very_wide) w.chunk32<16>(r, j0 + c);
          else w.chunk32<8>(r, j0 + c);
          c += 32;
        } else {
          uint32_t r[8];
          tmem_ld8(s_tmem + c, r);
          tmem_wait_ld();
          w.chunk8(r, j0 + c);
          c += 8;
        }
        __syncwarp();
      }
      ref = j0 + kWtKeys;
      tc_fence_before();
      mbar_arrive(bar_s_empty + 8 * slot);
    }
    // the row's last run: a1 is relative to the last visible key of the part
    if (w.cur >= 0) w.flush(w.weight(min(ref - 1, w.i)));
    row_l = w.l; row_base = w.base;
    fac_s[g * 128 + row] = w.base;
    first_s[g * 128 + row] = w.first;
  }
  __syncthreads();
  // ---- the parts of a row: a common base, the sum of all, the factor that normalises each part's bins
  const int at = ((warp - 2) >> 2) * 128 + (warp & 3) * 32 + lane, row = at & 127;   // epilogue threads: [part][row]
  auto all_parts = [&](auto f) { return f(f(fac_s[row], fac_s[128 + row]), f(fac_s[256 + row], fac_s[384 + row])); };
  static_assert(kWtParts == 4, "all_parts");
  float factor = 0.f;
  if (warp >= 2) {
    const float m = all_parts([](float a, float b) { return fmaxf(a, b); });
    factor = (row_base == -INFINITY) ? 0.f : ex2_approx((row_base - m) * (p.scale * 1.44269504f));
  }
  __syncthreads();
  if (warp >= 2) fac_s[at] = row_l * factor;
  __syncthreads();
  if (warp >= 2) {
    const float l = all_parts([](float a, float b) { return a + b; });
    factor = i0 + row < p.n ? __fdiv_rn(factor, l) : 0.f;
    aside_s[at] = first_s[at] >= 0 ? aside_s[at] * factor : 0.f;
  }
  __syncthreads();
  if (warp >= 2) fac_s[at] = factor;
  __syncthreads();
  if (*cta_abort) {
    const uint64_t t_wait = globaltimer_ns();   // copies may still be in flight towards this CTA's shared memory
    while (globaltimer_ns() - t_wait < 200000ull) __nanosleep(1000);
    poison();
  } else {
    // ---- a warp per bin: the 128 rows' values, each with the factor of the part that stored it: the last one whose
    // first bin lies above
    float fac[kWtParts][4], aside[kWtParts][4];
    int first[kWtParts][4];
#pragma unroll
    for (int g = 0; g < kWtParts; ++g)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = g * 128 + lane + 32 * u;
        fac[g][u] = fac_s[e]; aside[g][u] = aside_s[e]; first[g][u] = first_s[e];
      }
    for (int b = warp; b < p.nbins; b += kWtThreads / 32) {
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float v = hist[b * 128 + lane + 32 * u];
        float f = fac[0][u];
#pragma unroll
        for (int g = 1; g < kWtParts; ++g) {
          if (b < first[g][u]) f = fac[g][u];
          if (b == first[g][u]) s += aside[g][u];
        }
        if (v != 0.f) s += v * f;   // a bin that no key of the row fell into stays out, whatever the factor (a NaN sum)
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0 && s != 0.f) atomicAdd(out + b, static_cast<double>(s));
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace sq
