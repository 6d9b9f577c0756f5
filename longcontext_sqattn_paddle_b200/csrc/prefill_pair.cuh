// Causal GQA prefill attention on 256-row query blocks: long dense causal and relative-window calls with one operand set and an
// f16 P (prefill.cuh holds the other cases; the rule is at the launch).
//
// One CTA per SM walks blocks of 256 query rows of one head: two 128-row tiles A and B on shared 128-key K / V tiles.
//   warp 0       TMA producer: two stages of K and two of V; the Q tiles of the next block
//   warp 1       tcgen05 issuer: P V and the next Q K^T of tile A, then the same of tile B; owns all 512 TMEM columns
//   warp 2       writes the issuer's program: one word per step, so that the issuer neither walks nor divides
//   warps 4..7   online softmax and epilogue of tile A, warps 8..11 of tile B: one query row per thread (TMEM lane)
// While one tile's 128 x 128 scores go through the softmax warps the tensor core works on the other tile.
//
// What bounds it: the 1 kW power limit.  A 256 x 128 step takes 3250 clocks (2048 of them on the tensor pipe) where two CTAs of
// prefill_kernel need 4060, but the clock settles at 1.37 GHz under load instead of 1.6 (dense 32768 tokens: 10.2 M clocks
// against 12.6 M, 7.04 ms against 7.23 in a loop, 6.27 against 6.38 after a pause).  What it saves is energy: K and V arrive in
// shared memory once for 256 rows, and a 128-key Q K^T reads Q half as often as two 64-key ones (prefill_kernel without its
// TMA loads: 0.9x the time, sustained).
// The issuer decides whether the tensor core is kept busy, whose queue is a few instructions deep: rolled loops (40-50 clocks
// an instruction instead of 12), a branch per instruction or the walk in this warp each cost as much as the softmax (9.6 ms).
#pragma once
#include "prefill.cuh"

namespace sq {

constexpr int kPairN = 128;      // keys per step
constexpr int kPairStages = 2;   // K tiles in shared memory, and V tiles
constexpr int kPairThreads = 384;
constexpr int kPairProg = 32;    // steps in one half of the issuer's program
// A step of the issuer's program: P V of a step and Q K^T of the one after it, for tile x
constexpr uint32_t kProgPv = 1, kProgHalves = 1 << 2, kProgFirstPv = 1 << 6, kProgLastPv = 1 << 8;   // << x (halves: << 2 x)
constexpr uint32_t kProgQk = 1 << 10, kProgFirstQk = 1 << 12, kProgLastQk = 1 << 14;                 // << x
constexpr uint32_t kProgEnd = 1 << 16;

template <int D>
struct PairSmem {
  static constexpr int kTile = 128 * D * 2;   // a Q, K or V tile
  static constexpr int kQOff = 0;
  static constexpr int kKOff = 2 * kTile;
  static constexpr int kVOff = kKOff + kPairStages * kTile;
  static constexpr int kBarOff = kVOff + kPairStages * kTile;
  // barriers: q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2], prog_full[2], prog_empty[2], s_full[2],
  // p_full[2][2] (64-key half, tile), o_full[2]
  static constexpr int kSingleBars = 8 + 4 * kPairStages;   // those that one arrival completes, ahead of the others
  static constexpr int kNumBars = kSingleBars + 8;
  static constexpr int kMiscOff = kBarOff + 8 * kNumBars;   // tmem base, abort flag
  static constexpr int kProgOff = kMiscOff + 16;
  static constexpr int kDynBytes = kProgOff + 2 * kPairProg * 4;
};

// The key tiles (128 keys from 128 t on) that a 256-row block visits.  Tile X in {A, B} of the block visits [0, s[X]) (the sink
// and what lies before the block) and [l[X], h[X]) (window and diagonal); both bounds grow from A to B.  The walk is ascending,
// so that a tile meets its keys in the same order whichever tile it is paired with, and says who takes part in a step.
struct PairBlock {
  int bi, head, kvh, row0;   // row0: local row of A's first row
  int g;                // 128-row block of A in the whole sequence
  int has_b;
  int s[2], l[2], h[2];
  int edge_s[2], edge_l[2], edge_h[2];   // which 64-key halves of tiles s - 1, l and h - 1 some row visits (of the others: both)
  __host__ __device__ void segment(int i, int& t0, int& t1, int& act) const {
    auto lesser = [](int a, int b) { return a < b ? a : b; };
    auto larger = [](int a, int b) { return a > b ? a : b; };
    act = i == 4 ? 1 : (i == 1 || i == 3 || i == 6 ? 2 : (has_b ? 3 : 1));
    switch (i) {
      case 0: t0 = 0; t1 = s[0]; break;
      case 1: t0 = s[0]; t1 = lesser(s[1], l[0]); break;
      case 2: t0 = l[0]; t1 = lesser(h[0], s[1]); break;
      case 3: t0 = h[0]; t1 = s[1]; break;
      case 4: t0 = larger(l[0], s[1]); t1 = lesser(l[1], h[0]); break;
      case 5: t0 = l[1]; t1 = h[0]; break;
      default: t0 = larger(l[1], h[0]); t1 = h[1]; break;
    }
  }
  __host__ __device__ int steps(int x) const { return s[x] + h[x] - l[x]; }
  __host__ __device__ int halves(int x, int t) const {
    return t == l[x] ? edge_l[x] : (t == s[x] - 1 ? edge_s[x] : (t == h[x] - 1 ? edge_h[x] : 3));
  }
};
constexpr int kPairSegs = 7;

// What the rows [qs, qe) of one block of the reference's loop see: keys [0, s), [lo, qs), and [qs, qe) causally.
struct RowView {
  int s, lo, qs, qe;
  // the 64 keys from k0 on: 0 = not visited, 1 = whole, 2 = on the diagonal
  __host__ __device__ int kind(int k0) const {
    if (k0 >= qs) return k0 < qe ? 2 : 0;
    return (k0 < s || k0 >= lo) ? 1 : 0;
  }
};
__host__ __device__ inline RowView row_view(const PrefillParams& p, int head, int g, int half) {
  RowView v;
  if (p.mode == 0) {   // dense: blocks of 128 rows
    v.qs = g * kBlockM; v.qe = v.qs + kBlockM; v.s = 0; v.lo = 0;
    return v;
  }
  v.qs = g * kBlockM + 64 * half;
  v.qe = v.qs + 64;
  if (v.qs >= p.n_total) {   // rows past the sequence visit nothing
    v.s = 0; v.lo = v.qs; v.qe = v.qs;
    return v;
  }
  int lo2, hi2, lo3, hi3;
  stage_range(2, v.qs, v.qe, p.w8[head], p.w4[head], p.sink, lo2, hi2);
  stage_range(3, v.qs, v.qe, p.w8[head], p.w4[head], p.sink, lo3, hi3);
  v.s = p.sink < v.qs ? p.sink : v.qs;
  v.lo = v.qs;
  if (hi3 > lo3) v.lo = lo3;
  if (hi2 > lo2 && lo2 < v.lo) v.lo = lo2;
  return v;
}

// Blocks of the launch in the order they are walked: the latest (for dense causal work: longest) first, heads fastest, so that
// the heads of a KV group share K and V through L2; the CTAs' order turns round every time, which evens out their work.
struct PairGrid {
  int n1, nblk2, per_blk;
  __host__ __device__ explicit PairGrid(const PrefillParams& p)
      : n1((p.blk_split + 1) / 2), nblk2(n1 + (p.nblk - p.blk_split + 1) / 2), per_blk(p.hq * p.batch) {}
  __host__ __device__ int items() const { return nblk2 * per_blk; }
  __host__ __device__ bool block(const PrefillParams& p, int cta, int ctas, int round, PairBlock& b) const {
    const int k = round * ctas + ((round & 1) ? ctas - 1 - cta : cta);
    if (k >= items()) return false;
    const int m = nblk2 - 1 - k / per_blk, rem = k % per_blk;
    b.bi = rem / p.hq; b.head = rem % p.hq; b.kvh = b.head / p.groups;
    const int local = m < n1 ? 2 * m : p.blk_split + 2 * (m - n1);
    b.has_b = local + 1 < (m < n1 ? p.blk_split : p.nblk);
    b.row0 = local * kBlockM;
    b.g = m < n1 ? p.blk0 + local : p.blk0_b + (local - p.blk_split);
    for (int x = 0; x < 2; ++x) {
      const RowView v0 = row_view(p, b.head, b.g + x, 0), v1 = row_view(p, b.head, b.g + x, 1);
      const int lo = v0.lo < v1.lo ? v0.lo : v1.lo, s = v0.s > v1.s ? v0.s : v1.s;
      b.s[x] = (s + kPairN - 1) / kPairN;
      b.l[x] = lo / kPairN > b.s[x] ? lo / kPairN : b.s[x];
      b.h[x] = b.g + x + 1;
      auto halves = [&](int k0) { return (v0.kind(k0) | v1.kind(k0) ? 1 : 0) | (v0.kind(k0 + 64) | v1.kind(k0 + 64) ? 2 : 0); };
      b.edge_s[x] = halves((b.s[x] - 1) * kPairN); b.edge_l[x] = halves(b.l[x] * kPairN); b.edge_h[x] = halves((b.h[x] - 1) * kPairN);
    }
    if (!b.has_b) { b.s[1] = b.s[0]; b.l[1] = b.l[0]; b.h[1] = b.h[0]; }
    return true;
  }
};

// Walks the steps of all blocks of a CTA.
struct PairWalk {
  const PrefillParams& p;
  PairGrid grid;
  PairBlock b;
  int round, seg, t, t1, act;
  bool valid;
  __device__ explicit PairWalk(const PrefillParams& p_) : p(p_), grid(p_), round(0), seg(-1), t(0), t1(0), act(0) {
    valid = grid.block(p, blockIdx.x, gridDim.x, 0, b);
    if (valid) settle();
  }
  __device__ void settle() {   // to the first tile at or after the present place
    while (t >= t1) {
      if (++seg == kPairSegs) {
        ++round;
        valid = grid.block(p, blockIdx.x, gridDim.x, round, b);
        if (!valid) return;
        seg = 0;
      }
      b.segment(seg, t, t1, act);
    }
  }
  __device__ void next() { ++t; settle(); }
};

template <int D>
__global__ void __launch_bounds__(kPairThreads, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ PrefillParams p) {
  using L = PairSmem<D>;
  constexpr uint32_t kTmemCols = 512;   // S_A [0,128) S_B [128,256) O_A [256,256+D) O_B [384,384+D); P over the first half of S
  constexpr uint32_t kOCol = 256;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  const uint32_t sbase = smem_u32(smem);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // the roles are uniform branches
  auto poison_all = [&]() {   // no block of this CTA can be trusted
    const PairGrid grid(p);
    PairBlock b;
    for (int round = 0; grid.block(p, blockIdx.x, gridDim.x, round, b); ++round) {
      poison_output<D>(p, b.bi, b.head, b.row0 / kBlockM);
      if (b.has_b) poison_output<D>(p, b.bi, b.head, b.row0 / kBlockM + 1);
    }
  };
  if ((sbase & 1023u) && threadIdx.x == 0) record_failure(130);
  if ((sbase & 1023u) || cta_device_failed()) {
    griddep_wait();
    poison_all();
    return;
  }
  const uint32_t q_s = sbase + L::kQOff, k_s = sbase + L::kKOff, v_s = sbase + L::kVOff, bars = sbase + L::kBarOff;
  const uint32_t bar_q_full = bars, bar_q_empty = bars + 16, bar_k_full = bars + 32, bar_k_empty = bars + 48;
  const uint32_t bar_v_full = bars + 64, bar_v_empty = bars + 80, bar_prog_full = bars + 96, bar_prog_empty = bars + 112;
  const uint32_t bar_s_full = bars + 128, bar_p_full = bar_s_full + 16, bar_o_full = bar_p_full + 32;
  volatile uint32_t* tmem_base_s = reinterpret_cast<volatile uint32_t*>(smem + L::kMiscOff);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  uint32_t* prog = reinterpret_cast<uint32_t*>(smem + L::kProgOff);
  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int i = 0; i < L::kSingleBars; ++i) mbar_init(bars + 8 * i, 1);
    for (int x = 0; x < 2; ++x) {
      mbar_init(bar_s_full + 8 * x, 1); mbar_init(bar_p_full + 8 * x, 4); mbar_init(bar_p_full + 16 + 8 * x, 4); mbar_init(bar_o_full + 8 * x, 1);
    }
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
  constexpr uint32_t tmem = 0;   // all 512 columns are this CTA's (checked below)
  const bool tmem_ok = *tmem_base_s == 0;
  griddep_wait();   // the set-up above may run while the kernel before this one drains
  if (!tmem_ok && threadIdx.x == 0) { record_failure(139); *cta_abort = 1; }

  if (!tmem_ok) {
  } else if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- TMA producer
      tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v);
      bool ok = true;
      uint32_t u = 0, nq[2] = {0, 0};   // steps, Q tiles loaded
      int round = -1;
      auto load = [&](const CUtensorMap* tm, uint32_t dst, uint32_t full, uint32_t empty, const PairWalk& w) {
        const uint32_t st = u & 1;
        if (u >= kPairStages) ok = mbar_wait(empty + 8 * st, (u / kPairStages - 1) & 1, cta_abort, 131);
        if (!ok) return;
        mbar_expect_tx(full + 8 * st, L::kTile);
#pragma unroll
        for (int h = 0; h < D / 64; ++h)
          tma_load_4d(dst + st * L::kTile + h * (kPairN * 128), tm, full + 8 * st, h * 64, w.t * kPairN, w.b.kvh, w.b.bi);
      };
      for (PairWalk w(p); ok && w.valid; w.next(), ++u) {
        load(&tm_k, k_s, bar_k_full, bar_k_empty, w);
        if (ok && w.round != round) {
          round = w.round;
          for (int x = 0; x < 1 + w.b.has_b; ++x) {
            if (nq[x] > 0) ok = ok && mbar_wait(bar_q_empty + 8 * x, (nq[x] - 1) & 1, cta_abort, 132);
            if (!ok) break;
            mbar_expect_tx(bar_q_full + 8 * x, L::kTile);
#pragma unroll
            for (int h = 0; h < D / 64; ++h)
              tma_load_4d(q_s + x * L::kTile + h * (kBlockM * 128), &tm_q, bar_q_full + 8 * x, h * 64, w.b.row0 + x * kBlockM, w.b.head, w.b.bi);
            ++nq[x];
          }
        }
        if (ok) load(&tm_v, v_s, bar_v_full, bar_v_empty, w);
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- tcgen05 issuer (converged warp, see prefill.cuh)
      const uint32_t fmt = p.qk_bf16 ? 1u : 0u;
      const uint32_t idesc_qk = make_idesc(fmt, fmt, 0, 0, kBlockM, kPairN);
      const uint32_t idesc_pv = make_idesc(0, 0, 0, 1, kBlockM, D);
      const uint64_t q_desc = smem_desc_sw128(q_s, 16, 1024);
      const uint64_t k_desc = smem_desc_sw128(k_s, 16, 1024);
      const uint64_t v_desc = smem_desc_sw128(v_s, kPairN * 128, 1024);
      bool ok = true;
      uint32_t q_par = 0, p_par = 0;   // bit x: phase of tile x's barrier
      uint32_t words = 0;              // lane j: step j of the present half of the program
      // A wait that gives up leaves through the loop's head: what is issued until then goes nowhere but tensor memory.
      auto await = [&](uint32_t bar, uint32_t parity, int code) {
        if (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) ok &= mbar_wait_warp(bar, parity, cta_abort, code);
      };
#pragma unroll 1
      for (uint32_t i = 0; ok; ++i) {
        // program step i: P V of step i - 1, Q K^T of step i
        if (i % kPairProg == 0) {
          await(bar_prog_full + 8 * (i / kPairProg & 1), (i / kPairProg >> 1) & 1, 140);
          if (!ok) break;
          words = prog[i % (2 * kPairProg) + lane];
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_prog_empty + 8 * (i / kPairProg & 1));
        }
        const uint32_t w = __shfl_sync(0xffffffffu, words, i % kPairProg);
        const uint32_t vst = (i - 1) & 1, kst = i & 1;
        const uint64_t vd = v_desc + (vst * L::kTile >> 4), kd = k_desc + (kst * L::kTile >> 4);
        // The tiles are looked at ahead of P, so that nothing stands between P's arrival and the sixteen products: the tensor
        // core's queue is only a few instructions deep.
        {
          const bool seen = (!(w & (3 * kProgPv)) || mbar_try_wait(bar_v_full + 8 * vst, ((i - 1) >> 1) & 1)) &
                            (!(w & (3 * kProgQk)) || mbar_try_wait(bar_k_full + 8 * kst, (i >> 1) & 1));
          if (!__all_sync(0xffffffffu, seen)) {
            if (w & (3 * kProgPv)) await(bar_v_full + 8 * vst, ((i - 1) >> 1) & 1, 135);
            if (w & (3 * kProgQk)) await(bar_k_full + 8 * kst, (i >> 1) & 1, 134);
          }
        }
#pragma unroll
        for (uint32_t x = 0; x < 2; ++x) {
          if (w & kProgFirstQk << x) {
            await(bar_q_full + 8 * x, (q_par >> x) & 1, 133);
            q_par ^= 1u << x;
          }
          if (w & kProgPv << x) {
            // O_x += P_x V over the 64-key halves that some row of the tile visits
            uint32_t acc = !(w & kProgFirstPv << x);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              await(bar_p_full + 16 * h + 8 * x, (p_par >> x) & 1, 136);
              tc_fence_after();
              if (w & kProgHalves << (2 * x + h)) {
#pragma unroll
                for (int kk = 4 * h; kk < 4 * h + 4; ++kk)
                  mma_ts_elect(tmem + kOCol + x * 128, tmem + x * kPairN + kk * 8, vd + (kk * 2048 >> 4), idesc_pv, (kk & 3) > 0 || acc);
                acc = 1;
              }
            }
            p_par ^= 1u << x;
          }
          if (w & kProgQk << x) {
            // S_x = Q_x K^T
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const uint32_t off = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
              mma_ss_elect(tmem + x * kPairN, q_desc + ((x * L::kTile + off) >> 4), kd + (off >> 4), idesc_qk, kk > 0);
            }
            tc_commit_elect(bar_s_full + 8 * x);
            if (w & kProgLastQk << x) tc_commit_elect(bar_q_empty + 8 * x);
          }
          if (w & kProgLastPv << x) tc_commit_elect(bar_o_full + 8 * x);
        }
        if (w & (3 * kProgPv)) tc_commit_elect(bar_v_empty + 8 * vst);
        if (w & (3 * kProgQk)) tc_commit_elect(bar_k_empty + 8 * kst);
        if (w & kProgEnd) break;
      }
    } else if (warp == 2 && lane == 0) {
      // ---------------------------------------------------------------- the issuer's program, two halves of kPairProg steps
      bool ok = true, end = false;
      int qk[2] = {0, 0}, pv[2] = {0, 0};   // steps of the present block
      PairWalk cur(p), nxt(p);
      for (uint32_t i = 0; ok && !end; ++i) {
        const uint32_t half = i / kPairProg;
        if (i % kPairProg == 0 && half >= 2) ok = mbar_wait(bar_prog_empty + 8 * (half & 1), (half / 2 - 1) & 1, cta_abort, 141);
        if (!ok) break;
        uint32_t w = 0;
        if (i > 0) {
          for (int x = 0; x < 2; ++x)
            if (cur.act >> x & 1) {
              w |= kProgPv << x | cur.b.halves(x, cur.t) * kProgHalves << 2 * x;
              if (pv[x] == 0) w |= kProgFirstPv << x;
              if (++pv[x] == cur.b.steps(x)) { pv[x] = 0; w |= kProgLastPv << x; }
            }
          cur.next();
        }
        if (nxt.valid) {
          for (int x = 0; x < 2; ++x)
            if (nxt.act >> x & 1) {
              w |= kProgQk << x;
              if (qk[x] == 0) w |= kProgFirstQk << x;
              if (++qk[x] == nxt.b.steps(x)) { qk[x] = 0; w |= kProgLastQk << x; }
            }
          nxt.next();
        }
        end = !cur.valid;
        if (end) w |= kProgEnd;
        prog[i % (2 * kPairProg)] = w;
        if (end || i % kPairProg == kPairProg - 1) mbar_arrive(bar_prog_full + 8 * (half & 1));
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int x = (warp >> 2) - 1;
    const int quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_tmem = tmem + lane_addr + x * kPairN, o_tmem = tmem + lane_addr + kOCol + x * 128;
    const uint32_t bar_s = bar_s_full + 8 * x, bar_p = bar_p_full + 8 * x, bar_o = bar_o_full + 8 * x;
    bool ok = true;
    uint32_t ns = 0, no = 0;   // steps and blocks so far
    PairWalk w(p);
    while (ok && w.valid) {
      const int round = w.round;
      const PairBlock b = w.b;
      const bool present = x == 0 || b.has_b;
      const RowView view = row_view(p, b.head, b.g + x, quarter >> 1);
      const int row = (b.g + x) * kBlockM + row_in_tile;
      float m_i = -INFINITY, base = -INFINITY, l_i = 1.0f;
      bool first = true;
      for (; ok && w.valid && w.round == round; w.next()) {
        if (!(w.act >> x & 1)) continue;
        ok = mbar_wait_warp(bar_s, ns & 1, cta_abort, 137);
        ++ns;
        if (!ok) break;
        tc_fence_after();
        uint32_t r0[64], r1[64];
        tmem_ld64(s_tmem, r0);
        tmem_ld64(s_tmem + 64, r1);
        tmem_wait_ld64(r0);
        tmem_ready64(r1);
        float s[128];
#pragma unroll
        for (int c = 0; c < 64; ++c) { s[c] = __uint_as_float(r0[c]); s[64 + c] = __uint_as_float(r1[c]); }
        const int k0 = w.t * kPairN;
        const int kind0 = view.kind(k0), kind1 = view.kind(k0 + 64);
        if ((kind0 & kind1) != 1) {   // an edge of the visited range or the diagonal
          const int last = row - k0;
          if (kind0 == 0) {
#pragma unroll
            for (int c = 0; c < 64; ++c) s[c] = -INFINITY;
          } else if (kind0 == 2) {
#pragma unroll
            for (int c = 0; c < 64; ++c) s[c] += c <= last ? 0.0f : -1000000.0f;
          }
          if (kind1 == 0) {
#pragma unroll
            for (int c = 64; c < 128; ++c) s[c] = -INFINITY;
          } else if (kind1 == 2) {
#pragma unroll
            for (int c = 64; c < 128; ++c) s[c] += c <= last ? 0.0f : -1000000.0f;
          }
        }
        // P and the row's sum of 32 keys, relative to `ref`
        uint64_t sums[2] = {f32x2_pack(0.f, 0.f), f32x2_pack(0.f, 0.f)};
        uint32_t pk[16];
        auto exponentials = [&](int q, float ref) {
          const uint64_t m2 = f32x2_pack(ref, ref);
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float u, v;
            f32x2_unpack(f32x2_sub(f32x2_pack(s[32 * q + c], s[32 * q + c + 1]), m2), u, v);
            u = ex2_approx(u); v = ex2_approx(v);
            sums[(c >> 1) & 1] = f32x2_add(sums[(c >> 1) & 1], f32x2_pack(u, v));
            pk[c >> 1] = pack_f16x2(u, v);
          }
        };
        // The lazy reference (prefill.cuh) rarely moves: the first 32 exponentials take it as it stands, beside the search for
        // the maximum, and are computed again where some row of the warp has moved.
        float ref = base == -INFINITY ? 0.0f : base;   // no key of this row visited yet: P = 0
        exponentials(0, ref);
        float mx[4] = {m_i, s[0], s[1], s[2]};
#pragma unroll
        for (int c = 3; c < 127; c += 2) mx[(c >> 1) & 3] = max3(mx[(c >> 1) & 3], s[c], s[c + 1]);
        const float m_new = fmaxf(max3(mx[0], mx[1], mx[2]), fmaxf(mx[3], s[127]));
        m_i = m_new;
        float alpha = 1.0f;
        const bool moved = m_new > base + kLazyLog2;
        if (__any_sync(0xffffffffu, moved)) {
          if (moved) { alpha = ex2_approx(base - m_new); base = m_new; }
          if (!first) {
            // P V of the step before has completed: it was issued ahead of the Q K^T this warp has waited for
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 16) {
              uint32_t o[16];
              tmem_ld16(o_tmem + c0, o);
              tmem_wait_ld();
              const uint64_t al2 = f32x2_pack(alpha, alpha);
#pragma unroll
              for (int c = 0; c < 16; c += 2) {
                float u, v;
                f32x2_unpack(f32x2_mul(f32x2_pack(__uint_as_float(o[c]), __uint_as_float(o[c + 1])), al2), u, v);
                o[c] = __float_as_uint(u); o[c + 1] = __float_as_uint(v);
              }
              tmem_st16(o_tmem + c0, o);
            }
          }
          ref = base == -INFINITY ? 0.0f : base;
          sums[0] = sums[1] = f32x2_pack(0.f, 0.f);
          exponentials(0, ref);
        }
        first = false;
        tmem_st16(s_tmem, pk);
#pragma unroll
        for (int q = 1; q < 4; ++q) {
          exponentials(q, ref);
          tmem_st16(s_tmem + q * 16, pk);
          if (q & 1) {   // 64 keys of P are handed over at a time: P V of the first half runs under the second's exponentials
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p + 16 * (q >> 1));
          }
        }
        float s0, s1, s2, s3;
        f32x2_unpack(sums[0], s0, s1);
        f32x2_unpack(sums[1], s2, s3);
        l_i = l_i * alpha + ((s0 + s1) + (s2 + s3));
      }
      if (!ok || !present) continue;
      ok = mbar_wait_warp(bar_o, no & 1, cta_abort, 138);
      ++no;
      if (!ok) break;
      tc_fence_after();
      const int row_local = b.row0 + x * kBlockM + row_in_tile;
      const bool in_range = row_local < p.n;
      uint8_t* orow = reinterpret_cast<uint8_t*>(p.o) +
                      2 * (static_cast<long long>(b.bi) * p.o_sb + static_cast<long long>(b.head) * p.o_sh +
                           static_cast<long long>(row_local) * p.o_sn);
      const float inv = 1.0f / l_i;
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        tmem_ld32(o_tmem + c0, o);
        tmem_wait_ld();
        if (in_range) {
          uint32_t wd[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const float u = __uint_as_float(o[2 * c]) * inv, v = __uint_as_float(o[2 * c + 1]) * inv;
            wd[c] = p.o_dtype ? pack_bf16x2(u, v) : pack_f16x2(u, v);
          }
          uint4* dst = reinterpret_cast<uint4*>(orow + c0 * 2);
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[c] = make_uint4(wd[4 * c], wd[4 * c + 1], wd[4 * c + 2], wd[4 * c + 3]);
        }
      }
      if (p.lse && in_range)
        p.lse[(static_cast<long long>(b.bi) * p.hq + b.head) * p.n + row_local] = log2f(l_i) + base;
      tc_fence_before();   // the next block's P V may overwrite O once this warp has handed over its first P
    }
  }

  // ------------------------------------------------------------------ tear-down (also reached after a wait gave up)
  if (*cta_abort) {
    // copies may still be in flight towards this CTA's shared memory: give them time to land
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (*cta_abort) poison_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace sq
