// Relative-distance attention-energy histogram (window_search.cuh states the rule) on the 5th-generation tensor cores,
// in ONE sweep over the keys of a row block.
//
// What bounds it: one exponential per (query, key) pair.  The mma.sync kernel swept the keys twice (statistics, then
// normalised weights), computed two exponentials and an IEEE division per pair and took 10.6 ms for 28 heads x 8192
// tokens x 200 bins (this one 1.85 ms); the products of one sweep are 0.15 ms of the measured tensor rate, its exponentials 0.2 ms of the
// special-function units.  Hence:
//   * a thread owns one query row (a TMEM lane) and meets its keys in order, so its bins never increase: a bin is one
//     run, kept as A0 = sum a and A1 = sum a * (j - ref) with a = 2^(score - base) NOT normalised, and stored once, in a
//     per-row histogram in shared memory; the row sum is known at the end and scales the stored bins then.  base is the
//     maximum of the row's first keys; fp32 holds a up to 2^60 above it, so it moves (and the stored bins are rescaled)
//     only past that.
//   * the bin of a key is not computed per pair: the run knows the first key of the next bin (next_key), from the fp32
//     expressions of the reference evaluated at a bin's edge.
//   * one CTA = 128 rows of one head.  The keys up to the diagonal are cut in two halves at a 128-key tile: epilogue
//     warps 2..5 walk the first half, warps 6..9 the second, each with two 128-column accumulators, so that eight warps
//     share the exponentials of a row block although the per-row histogram (nbins x 128 fp32) leaves room for one CTA.
//     The bin in which the halves meet is the only one that both write; the second half keeps its part aside.
//   warp 0 TMA producer, warp 1 tcgen05 issuer (owns the 512 TMEM columns).
#pragma once
#include <cuda.h>

#include "ptx.cuh"
#include "window_search.cuh"

namespace sq {

constexpr int kWtRows = 128, kWtKeys = 128;
constexpr int kWtMaxBins = 256;       // nbins x 128 fp32 + Q tile + one K stage per half within 227 KB
constexpr int kWtKeysPerBin = 1024;   // seq_len / nbins at most this: see next_key
constexpr int kWtFastWidth = 9;       // bins at least this wide (keys): at most one edge among eight consecutive keys
constexpr float kWtLazyLog2 = 60.0f;

template <int D>
struct WindowTcSmem {
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kTileBytes;                  // one stage per half
  static constexpr int kRowOff = kKOff + 2 * kTileBytes;    // [2 halves][128] factor, [128] first bin, [128] its value
  static constexpr int kBarOff = kRowOff + 4 * 128 * 4;     // q_full, k_full[2], s_full[2][2], s_empty[2][2]
  static constexpr int kMiscOff = kBarOff + 8 * 11;
  static constexpr int kHistOff = kMiscOff + 24;            // 16-byte aligned; [nbins][128]
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
  float ctx, cinv, width;    // max(i - sink, 1); bins per key and keys per bin (0 and unused for rows without bins)
  float c2;                  // scores are raw dot products: exp(s * scale) = 2^(s * c2)
  float* hist;               // this row's column of [nbins][128]
  float base;                // raw score that the weights are relative to; -inf: no key yet
  float a0, a1, l;           // the current run (a1 relative to the current chunk's first key), sum of the finished runs
  int cur, next;             // bin of the current run (-1: none yet), first key behind it
  int first;                 // second half: its first bin, kept in first_val; -1 in the first half: every run is stored
  float first_val;
  bool keep_first;

  __device__ __forceinline__ int exact_bin(int dist) const {   // the reference's fp32 expressions (window_search.py:262-272)
    const float rel = (i <= sink) ? 0.f : __fdiv_rn(static_cast<float>(dist), ctx);
    return min(max(static_cast<int>(floorf(__fmul_rn(rel, static_cast<float>(nbins)))), 0), nbins - 1);
  }
  // First key whose bin is below b, given that b's edge lies at distance b * ctx / nbins: the smallest distance with
  // exact_bin >= b is one of the two integers around it.  Both the estimate and the reference's expression are within
  // 3e-5 bins of the true quotient and neighbouring distances at least 1 / kWtKeysPerBin bins apart, so only a distance
  // within 1e-4 bins of the edge needs the reference's expression itself.
  __device__ __forceinline__ int next_key(int b) const {
    if (b <= 0) return 0x7fffffff;
    const float fb = static_cast<float>(b);
    const float d0 = rintf(fb * width), off = __fmaf_rn(d0, cinv, -fb);
    int d = static_cast<int>(d0);
    if (fabsf(off) < 1e-4f) d += exact_bin(d) >= b ? 0 : 1;
    else d += off > 0.f ? 0 : 1;
    return i - d + 1;
  }
  __device__ __forceinline__ void flush(int c0) {
    const float t0 = __fmaf_rn(static_cast<float>(i - c0), cinv, 1.0f);
    const float w = __fmaf_rn(a0, t0, -cinv * a1);
    if (keep_first) { first = cur; first_val = w; keep_first = false; }
    else hist[cur * 128] = w;
    l += a0;
  }
  __device__ __forceinline__ void rebase(float mx) {
    if (base != -INFINITY) {
      const float f = ex2_approx((base - mx) * c2);
      a0 *= f; a1 *= f; l *= f; first_val *= f;
      const int end = first >= 0 ? first : (keep_first ? 0 : nbins);
      if (cur >= 0)
        for (int b = cur + 1; b < end; ++b) hist[b * 128] *= f;
    }
    base = mx;
  }
  __device__ __forceinline__ void look_at_max(float mx) {
    if (mx > base && (base == -INFINITY || (mx - base) * c2 > kWtLazyLog2)) rebase(mx);
  }
  __device__ __forceinline__ float shift() const { return base == -INFINITY ? 0.f : -(base * c2); }

  // 32 keys from c0 on, all of them visible and behind the sink, bins at least kWtFastWidth wide
  __device__ __forceinline__ void chunk32(const uint32_t (&r)[32], int c0) {
    float mx = max3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
#pragma unroll
    for (int c = 3; c < 31; c += 2) mx = max3(mx, __uint_as_float(r[c]), __uint_as_float(r[c + 1]));
    mx = fmaxf(mx, __uint_as_float(r[31]));
    look_at_max(mx);
    const float sh = shift();
    if (cur < 0) { cur = exact_bin(i - c0); next = next_key(cur); }
#pragma unroll
    for (int s = 0; s < 32; s += 8) {
      const int nb = next - c0;
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = ex2_approx(__fmaf_rn(__uint_as_float(r[s + e]), c2, sh));
      if (__any_sync(0xffffffffu, nb < s + 8)) {
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (s + e < nb) { a0 += x[e]; a1 = __fmaf_rn(x[e], static_cast<float>(s + e), a1); }
          else { v0 += x[e]; v1 = __fmaf_rn(x[e], static_cast<float>(s + e), v1); }
        }
        if (nb < s + 8) {
          flush(c0);
          a0 = v0; a1 = v1;
          next = next_key(--cur);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) { a0 += x[e]; a1 = __fmaf_rn(x[e], static_cast<float>(s + e), a1); }
      }
    }
    a1 = __fmaf_rn(-32.0f, a0, a1);
  }
  // 8 keys from c0 on, any of them past the row or in the sink, bins of any width
  __device__ __forceinline__ void chunk8(const uint32_t (&r)[8], int c0) {
    if (c0 > i) return;
    float mx = __uint_as_float(r[0]);
#pragma unroll
    for (int e = 1; e < 8; ++e) mx = (c0 + e <= i) ? fmaxf(mx, __uint_as_float(r[e])) : mx;
    look_at_max(mx);
    const float sh = shift();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = c0 + e;
      if (j > i) continue;
      const float x = ex2_approx(__fmaf_rn(__uint_as_float(r[e]), c2, sh));
      if (j < sink) { l += x; continue; }
      if (cur < 0 || j >= next) {
        if (cur >= 0) flush(c0);
        a0 = a1 = 0.f;
        cur = exact_bin(i - j);
        next = next_key(cur);
      }
      a0 += x;
      a1 = __fmaf_rn(x, static_cast<float>(e), a1);
    }
    a1 = __fmaf_rn(-8.0f, a0, a1);
  }
};

template <int D>
__global__ void __launch_bounds__(320, 1)
window_hist_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ WindowHistParams p, int bf16) {
  using L = WindowTcSmem<D>;
  constexpr uint32_t kTmemCols = 512;   // accumulator u of half g: columns (2 g + u) * 128
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
  if ((sbase & 1023u) || device_failed()) {
    if ((sbase & 1023u) && threadIdx.x == 0) record_failure(500);
    poison();
    return;
  }
  const uint32_t q_s = sbase + L::kQOff, k_s = sbase + L::kKOff, bars = sbase + L::kBarOff;
  const uint32_t bar_q = bars, bar_k = bars + 8, bar_s_full = bars + 24, bar_s_empty = bars + 56;   // [g], [2 g + u]
  volatile uint32_t* tmem_base_s = reinterpret_cast<volatile uint32_t*>(smem + L::kMiscOff);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  float* fac_s = reinterpret_cast<float*>(smem + L::kRowOff);           // [2][128]: base, then the bins' factor
  int* first_s = reinterpret_cast<int*>(smem + L::kRowOff + 1024);
  float* fval_s = reinterpret_cast<float*>(smem + L::kRowOff + 1536);
  float* hist = reinterpret_cast<float*>(smem + L::kHistOff);
  const int ntiles = blk + 1, n0 = ntiles / 2;                          // tiles of the first half
  const int n1 = ntiles - n0;                                           // ... of the second: n0 or n0 + 1

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int b = 0; b < 7; ++b) mbar_init(bars + 8 * b, 1);
    for (int b = 7; b < 11; ++b) mbar_init(bars + 8 * b, 128);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_base_s)), kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  for (int c = threadIdx.x; c < p.nbins * 32; c += 320) reinterpret_cast<uint4*>(hist)[c] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s;

  float row_l = 0.f, row_base = -INFINITY;   // of an epilogue thread's half row, for the combination below
  int row_first = -1;
  float row_fval = 0.f;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k);
      mbar_expect_tx(bar_q, L::kTileBytes);
#pragma unroll
      for (int h = 0; h < D / 64; ++h) tma_load_4d(q_s + h * (128 * 128), &tm_q, bar_q, h * 64, i0, head, 0);
      bool ok = true;
      for (int u = 0; ok && u < n1; ++u)
        for (int g = 0; ok && g < 2; ++g) {
          if (g == 0 && u >= n0) continue;
          // the half's stage was last read by the products of its tile u - 1
          if (u >= 1) ok = mbar_wait(bar_s_full + 8 * (2 * g + ((u - 1) & 1)), ((u - 1) >> 1) & 1, cta_abort, 501);
          if (!ok) break;
          mbar_expect_tx(bar_k + 8 * g, L::kTileBytes);
#pragma unroll
          for (int h = 0; h < D / 64; ++h)
            tma_load_4d(k_s + g * L::kTileBytes + h * (128 * 128), &tm_k, bar_k + 8 * g, h * 64, (g * n0 + u) * kWtKeys, kvh, 0);
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ tcgen05 issuer (converged warp, one elected lane)
    const uint32_t fmt = bf16 ? 1u : 0u;
    const uint32_t idesc = make_idesc(fmt, fmt, 0, 0, 128, kWtKeys);
    const uint64_t q_desc = smem_desc_sw128(q_s, 16, 1024);
    bool ok = mbar_wait_warp(bar_q, 0, cta_abort, 511);
    for (int u = 0; ok && u < n1; ++u)
      for (int g = 0; ok && g < 2; ++g) {
        if (g == 0 && u >= n0) continue;
        ok = mbar_wait_warp(bar_k + 8 * g, u & 1, cta_abort, 512);
        if (ok && u >= 2) ok = mbar_wait_warp(bar_s_empty + 8 * (2 * g + (u & 1)), ((u - 2) >> 1) & 1, cta_abort, 513);
        if (!ok) break;
        tc_fence_after();
        const uint64_t k_desc = smem_desc_sw128(k_s + g * L::kTileBytes, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * (128 * 128) + (kk & 3) * 32) >> 4;
          mma_ss_elect(tmem + (2 * g + (u & 1)) * kWtKeys, q_desc + off, k_desc + off, idesc, kk > 0);
        }
        tc_commit_elect(bar_s_full + 8 * (2 * g + (u & 1)));
      }
  } else {
    // ------------------------------------------------------------------ epilogue: one row per thread, half g of its keys
    const int g = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int i_first = i0 + quarter * 32;                              // the warp's first row
    WindowRow w;
    w.i = i0 + row < p.n ? i0 + row : -1;                               // rows past the end see no key
    w.sink = p.sink; w.nbins = p.nbins;
    w.ctx = fmaxf(static_cast<float>(w.i - p.sink), 1.0f);
    w.cinv = w.i <= p.sink ? 0.f : __fdiv_rn(static_cast<float>(p.nbins), w.ctx);
    w.width = __fdiv_rn(w.ctx, static_cast<float>(p.nbins));
    w.c2 = p.scale * 1.44269504f;
    w.hist = hist + row;
    w.base = -INFINITY; w.a0 = w.a1 = w.l = 0.f; w.cur = -1; w.next = 0x7fffffff;
    w.first = -1; w.first_val = 0.f; w.keep_first = g == 1;
    const bool wide = i_first + 31 < p.n && i_first - p.sink >= kWtFastWidth * p.nbins;
    bool ok = true;
    int ref = 0;                                                        // key that a1 is relative to
    for (int u = 0; u < (g ? n1 : n0); ++u) {
      const uint32_t slot = 2 * g + (u & 1);
      ok = mbar_wait_warp(bar_s_full + 8 * slot, (u >> 1) & 1, cta_abort, 521);
      if (!ok) break;
      tc_fence_after();
      const uint32_t s_tmem = tmem + lane_addr + slot * kWtKeys;
      const int j0 = (g * n0 + u) * kWtKeys;
      if (wide && j0 >= p.sink && j0 + kWtKeys - 1 <= i_first) {
        uint32_t r0[32], r1[32];
        tmem_ld32(s_tmem, r0);
#pragma unroll 1
        for (int c = 0; c < kWtKeys; c += 64) {
          tmem_wait_ld();
          tmem_ld32(s_tmem + c + 32, r1);
          w.chunk32(r0, j0 + c);
          __syncwarp();
          tmem_wait_ld();
          if (c + 64 < kWtKeys) tmem_ld32(s_tmem + c + 64, r0);
          w.chunk32(r1, j0 + c + 32);
          __syncwarp();
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < kWtKeys; c += 8) {
          uint32_t r[8];
          tmem_ld8(s_tmem + c, r);
          tmem_wait_ld();
          w.chunk8(r, j0 + c);
          __syncwarp();
        }
      }
      ref = j0 + kWtKeys;
      tc_fence_before();
      mbar_arrive(bar_s_empty + 8 * slot);
    }
    // the row's last run: a1 is relative to the key behind the last chunk that was not skipped
    if (w.cur >= 0) w.flush(min(ref, (w.i & ~7) + 8));
    row_l = w.l; row_base = w.base; row_first = w.first; row_fval = w.first_val;
    fac_s[g * 128 + row] = w.base;
    if (g == 1) first_s[row] = w.first;
  }
  __syncthreads();
  // ---- the two halves of a row: a common base, the sum of both, the factor that normalises each half's bins
  const int g_row = (warp - 2) >> 2, row = (warp & 3) * 32 + lane;
  float factor = 0.f;
  if (warp >= 2) {
    const float m = fmaxf(fac_s[row], fac_s[128 + row]);
    const float c2 = p.scale * 1.44269504f;
    factor = (row_base == -INFINITY) ? 0.f : ex2_approx((row_base - m) * c2);
    row_l *= factor;
  }
  __syncthreads();
  if (warp >= 2) fac_s[g_row * 128 + row] = row_l;
  __syncthreads();
  if (warp >= 2) {
    const float l = fac_s[row] + fac_s[128 + row];
    const bool seen = i0 + row < p.n;
    factor = seen ? __fdiv_rn(factor, l) : 0.f;
    if (g_row == 1) fval_s[row] = row_first >= 0 ? row_fval * factor : 0.f;
  }
  __syncthreads();
  if (warp >= 2) fac_s[g_row * 128 + row] = factor;
  __syncthreads();
  if (*cta_abort) {
    const uint64_t t_wait = globaltimer_ns();   // copies may still be in flight towards this CTA's shared memory
    while (globaltimer_ns() - t_wait < 200000ull) __nanosleep(1000);
    poison();
  } else {
    // ---- a warp per bin: the 128 rows' values, each with the factor of the half that stored it
    float fa[4], fb[4], fv[4];
    int first[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      fa[u] = fac_s[lane + 32 * u]; fb[u] = fac_s[128 + lane + 32 * u];
      fv[u] = fval_s[lane + 32 * u]; first[u] = first_s[lane + 32 * u];
    }
    for (int b = warp; b < p.nbins; b += 10) {
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float v = hist[b * 128 + lane + 32 * u];
        // a bin that no key of the row fell into stays out, whatever the factor (a row whose sum is NaN)
        if (v != 0.f) s += v * (b >= first[u] ? fa[u] : fb[u]);
        if (b == first[u]) s += fv[u];
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
