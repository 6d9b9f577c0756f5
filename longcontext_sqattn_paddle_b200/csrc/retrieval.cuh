// Centroid-scored retrieval for clustered decode (the step the reference's logs hint at but its code lacks):
// score every cluster by <mean query of the KV group, centroid>, take clusters in descending score until a
// token budget is covered, emit the selected token indices in ascending order, gather their K/V rows.
// Scores are fp64 (exact products of 16-bit centroids and an fp32 mean, index-order sum), the selection is a search
// for the score at which the budget is covered, lowest index first among equal scores, so the selected indices are
// bit-exact and timing-independent.
#pragma once
#include "prep.cuh"

namespace sq {

constexpr int kRetMaxClusters = 4096;
constexpr int kRetMaxTokens = 262144;

struct RetrieveParams {
  const uint8_t* q;         // [G, groups, D] 16-bit
  const uint8_t* cent;      // [G, K, D] 16-bit
  const int* cluster_size;  // [G, K]
  const int* clusters;      // [G, K, max_cluster_size]
  int* out_idx;             // [G, cap]
  int* out_count;           // [G]
  int groups, num_clusters, d, max_cluster_size, num_tokens, budget, cap;
  int tail_start;           // tokens [tail_start, num_tokens) are not clustered yet (appended since the last fold) and
                            // are always selected; tail_start == num_tokens: none
};

template <bool BF16>
__device__ __forceinline__ void retrieve_select_body(const RetrieveParams& p, const int g) {
  extern __shared__ __align__(16) uint8_t rs[];
  double* scores = reinterpret_cast<double*>(rs);                                   // [K]
  uint32_t* bitmap = reinterpret_cast<uint32_t*>(rs + sizeof(double) * p.num_clusters);  // [ceil(T/32)]
  __shared__ float q_mean[128];
  __shared__ unsigned long long red_lo[32], red_hi[32];
  __shared__ int digit_w[256], digit_n[256];
  __shared__ int sel_list[kRetMaxClusters];
  __shared__ int n_sel, warp_sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.num_clusters, D = p.d;
  const uint16_t* q = reinterpret_cast<const uint16_t*>(p.q) + static_cast<long long>(g) * p.groups * D;
  const uint16_t* cent = reinterpret_cast<const uint16_t*>(p.cent) + static_cast<long long>(g) * K * D;
  const int* csize = p.cluster_size + static_cast<long long>(g) * K;
  const int* cl = p.clusters + static_cast<long long>(g) * K * p.max_cluster_size;
  const int words = (p.num_tokens + 31) / 32;

  if (tid < D) {  // mean query of the group: fp32, heads added in order
    float s = 0.f;
    for (int h = 0; h < p.groups; ++h) s += to_f32<BF16>(q[h * D + tid]);
    q_mean[tid] = s / static_cast<float>(p.groups);
  }
  for (int w = tid; w < words; w += blockDim.x) bitmap[w] = 0u;
  if (tid == 0) n_sel = 0;
  __syncthreads();
  // Scores: D/8 lanes per centroid row, 16-byte loads (a warp reads whole rows, coalesced), four rows per lane in
  // flight; each lane adds its eight products in index order, the lanes' sums are combined pairwise in a fixed
  // order, so a score does not depend on timing (and centroids with identical rows get identical scores).
  {
    const int lanes_per_row = D / 8, rows_per_warp = 32 / lanes_per_row;
    const int sub = lane % lanes_per_row, rslot = lane / lanes_per_row;
    constexpr int kInFlight = 4;
    // Conversions to fp64 run at a quarter of the fp64 rate: the centroids go in with their own exponent field and the
    // query carries the power of two that is missing (selection 29.2 -> 24.1 us for 8 sequences x 8 KV heads x 1024 centroids).
    double qd[8], qw[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      qd[e] = static_cast<double>(q_mean[sub * 8 + e]);
      qw[e] = qd[e] * narrow_scale<BF16>();
    }
    const int stride = (blockDim.x >> 5) * rows_per_warp;
    const int o1 = lanes_per_row >> 1, o2 = lanes_per_row >> 2;
    for (int c0 = warp * rows_per_warp; c0 < K; c0 += kInFlight * stride) {
      uint4 raw[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int c = c0 + u * stride + rslot;
        raw[u] = (c < K) ? *reinterpret_cast<const uint4*>(cent + static_cast<long long>(c) * D + sub * 8) : make_uint4(0, 0, 0, 0);
      }
      double sc[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        bool special = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) special |= narrow_special<BF16>(w[e]);
        sc[u] = 0.0;
        if (!special) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            sc[u] = fma(narrow_as_double<BF16>(w[e] & 0xffffu), qw[2 * e], sc[u]);
            sc[u] = fma(narrow_as_double<BF16>(w[e] >> 16), qw[2 * e + 1], sc[u]);
          }
        } else {
          float f[8];
          unpack8<BF16>(raw[u], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) sc[u] += static_cast<double>(f[e]) * qd[e];
        }
      }
      // The lanes' sums, pairs o1 lanes apart first, then o2 and so on, four rows at a time: each exchange halves the rows a
      // lane holds, and row (b1 ? 1 : 0) + (b2 ? 2 : 0) is left with it.
      static_assert(kInFlight == 4, "two exchanges");
      const bool b1 = sub & o1, b2 = sub & o2;
      const double k0 = (b1 ? sc[1] : sc[0]) + __shfl_xor_sync(0xffffffffu, b1 ? sc[0] : sc[1], o1);
      const double k1 = (b1 ? sc[3] : sc[2]) + __shfl_xor_sync(0xffffffffu, b1 ? sc[2] : sc[3], o1);
      double s = (b2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b2 ? k0 : k1, o2);
      for (int o = o2 >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int c = c0 + ((b1 ? 1 : 0) + (b2 ? 2 : 0)) * stride + rslot;
      if (c < K && (sub & (o2 - 1)) == 0) scores[c] = (csize[c] > 0) ? s : -1.0 / 0.0;  // empty clusters are never taken
    }
  }
  __syncthreads();
  // Selection: clusters in descending score (ties: lowest index) until their sizes cover the budget.  Only the SET is
  // needed, so nothing is sorted: the scores become 64-bit integers of the same order (0 = empty, below every real
  // score) and the key of the cluster that crosses the budget is found digit by digit, a histogram of the sizes per
  // digit value each time; a digit that a single cluster is left in ends the search.  Scores of one group share their
  // leading bits: the first digit starts at the highest bit in which the largest and the smallest key differ.
  // (Taking the best remaining cluster in rounds of two barriers each cost a round per cluster taken: a step of 8
  // sequences, 8 KV heads and a budget of 4096 tokens went from 140 to 88 us; this kernel is 24 us of its 68 now.)
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(scores);
  {
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int c = tid; c < K; c += blockDim.x) {
      const double v = scores[c];
      const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
      const unsigned long long k = (v == -1.0 / 0.0) ? 0ull : ((bits >> 63) ? ~bits : (bits | 0x8000000000000000ull));
      keys[c] = k;
      if (k) { lo = k < lo ? k : lo; hi = k > hi ? k : hi; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
      lo = l2 < lo ? l2 : lo; hi = h2 > hi ? h2 : hi;
    }
    if (lane == 0) { red_lo[warp] = lo; red_hi[warp] = hi; }
  }
  __syncthreads();
  unsigned long long thr;        // keys >= thr are taken ...
  int tie_need = 0;              // ... of those equal to thr, when this is positive, the first in index order until their
                                 // sizes cover so many tokens
  {
    unsigned long long lo = lane < static_cast<int>(blockDim.x >> 5) ? red_lo[lane] : ~0ull;
    unsigned long long hi = lane < static_cast<int>(blockDim.x >> 5) ? red_hi[lane] : 0ull;
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
      lo = l2 < lo ? l2 : lo; hi = h2 > hi ? h2 : hi;
    }
    // bits [shift, 64) of the crossing key are `prefix`; all candidates agree with it there
    int shift = hi == 0ull ? 0 : 64 - __clzll(static_cast<long long>(lo ^ hi));
    unsigned long long prefix = shift >= 64 ? 0ull : hi >> shift;
    int need = p.budget;
    thr = 1ull;                  // no key at all, or all of them together below the budget
    bool single = hi == 0ull;
    while (!single && shift > 0) {
      const int width = shift < 8 ? shift : 8, low = shift - width;
      if (tid < 256) { digit_w[tid] = 0; digit_n[tid] = 0; }
      __syncthreads();
      for (int c = tid; c < K; c += blockDim.x) {
        const unsigned long long k = keys[c];
        if (k != 0ull && (shift >= 64 || (k >> shift) == prefix)) {
          const int dg = static_cast<int>((k >> low) & ((1ull << width) - 1));
          atomicAdd(&digit_w[dg], csize[c]);
          atomicAdd(&digit_n[dg], 1);
        }
      }
      __syncthreads();
      // every warp finds the digit for itself: lane l holds the values 8 l .. 8 l + 7
      int w8[8], sum = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) { w8[u] = digit_w[lane * 8 + u]; sum += w8[u]; }
      int above = sum;           // sizes in this lane's digits and all higher ones
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(0xffffffffu, above, o);
        if (lane + o < 32) above += v;
      }
      const unsigned cross = __ballot_sync(0xffffffffu, above >= need);
      if (cross == 0u) { single = true; break; }   // first digit only: every key is taken (thr = 1)
      const int src = 31 - __clz(cross);
      int run = above - sum, dg = 0;
#pragma unroll
      for (int u = 7; u >= 0; --u) {
        if (run < need && run + w8[u] >= need) { dg = lane * 8 + u; sum = run; }
        run += w8[u];
      }
      dg = __shfl_sync(0xffffffffu, dg, src);
      need -= __shfl_sync(0xffffffffu, sum, src);
      prefix = (prefix << width) | static_cast<unsigned>(dg);
      shift = low;
      thr = prefix << shift;
      single = digit_n[dg] == 1;
      __syncthreads();           // the histogram is cleared next
    }
    if (!single && hi != 0ull) { thr = prefix; tie_need = need; }
  }
  if (tie_need == 0) {
    for (int c = tid; c < K; c += blockDim.x)
      if (keys[c] >= thr) sel_list[atomicAdd(&n_sel, 1)] = c;
  } else {
    for (int c = tid; c < K; c += blockDim.x)
      if (keys[c] > thr) sel_list[atomicAdd(&n_sel, 1)] = c;
    __syncthreads();
    if (warp == 0) {             // clusters of equal score, in index order
      int got = 0, n = n_sel;
      for (int c0 = 0; c0 < K && got < tie_need; c0 += 32) {
        const bool tied = c0 + lane < K && keys[c0 + lane] == thr;
        const int sz = tied ? csize[c0 + lane] : 0;
        int before = sz;
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, before, o);
          if (lane >= o) before += v;
        }
        const bool take = tied && got + before - sz < tie_need;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) sel_list[n + __popc(m & ((1u << lane) - 1u))] = c0 + lane;
        n += __popc(m);
        got += __shfl_sync(0xffffffffu, before, 31);
      }
      if (lane == 0) n_sel = n;
    }
  }
  __syncthreads();
  // members of the selected clusters -> bitmap over token positions
  const int ns = n_sel;
  for (int s = warp; s < ns; s += (blockDim.x >> 5)) {
    const int c = sel_list[s];
    const int n = min(csize[c], p.max_cluster_size);
    for (int j = lane; j < n; j += 32) {
      const int tok = cl[static_cast<long long>(c) * p.max_cluster_size + j];
      atomicOr(&bitmap[tok >> 5], 1u << (tok & 31));
    }
  }
  __syncthreads();
  // tokens appended since the clusters were last rebuilt: always attended
  for (int tok = p.tail_start + tid; tok < p.num_tokens; tok += blockDim.x) atomicOr(&bitmap[tok >> 5], 1u << (tok & 31));
  __syncthreads();
  // ordered compaction: each thread owns a contiguous run of bitmap words
  const int per = (words + blockDim.x - 1) / blockDim.x;
  const int w0 = min(words, tid * per), w1 = min(words, w0 + per);
  int cnt = 0;
  for (int w = w0; w < w1; ++w) cnt += __popc(bitmap[w]);
  int incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int v = warp_sums[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sums[lane] = v;
  }
  __syncthreads();
  int pos = incl - cnt + (warp > 0 ? warp_sums[warp - 1] : 0);
  int* out = p.out_idx + static_cast<long long>(g) * p.cap;
  for (int w = w0; w < w1; ++w) {
    uint32_t bits = bitmap[w];
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1;
      if (pos < p.cap) out[pos] = w * 32 + b;
      ++pos;
    }
  }
  if (tid == blockDim.x - 1) p.out_count[g] = min(pos, p.cap);
}

template <bool BF16>
__global__ void __launch_bounds__(1024) retrieve_select_kernel(const __grid_constant__ RetrieveParams p) {
  retrieve_select_body<BF16>(p, blockIdx.x);
}

// All sequences of a ragged batch in one launch: blockIdx.y = sequence, blockIdx.x = KV group.
constexpr int kRetMaxBatch = 32;
struct RetrieveBatch {
  RetrieveParams item[kRetMaxBatch];
};
template <bool BF16>
__global__ void __launch_bounds__(1024) retrieve_select_batch_kernel(const __grid_constant__ RetrieveBatch b) {
  retrieve_select_body<BF16>(b.item[blockIdx.y], blockIdx.x);
}

struct GatherItem {
  const uint8_t* src;   // [G, tokens, D] through strides
  uint8_t* dst;         // [G, cap, D]
  const int* idx;       // [G, cap]
  const int* count;     // [G]
  long long src_group_stride, src_row_stride;
  // block-hybrid caches: rows from split_row on live in a second buffer (pinned host memory, read over PCIe by the
  // same 16-byte loads), row r of it being token split_row + r; src2 == nullptr: everything is in src
  const uint8_t* src2;
  long long src2_group_stride;
  int split_row;
};
struct GatherBatch {
  GatherItem item[2 * kRetMaxBatch];  // keys and values of every sequence
};
__global__ void gather_rows_batch_kernel(const __grid_constant__ GatherBatch b, int cap, int d) {
  const GatherItem& it = b.item[blockIdx.z];
  const int g = blockIdx.y, d8 = d / 8;
  const int n = it.count[g];
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < static_cast<long long>(n) * d8;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i / d8), c = static_cast<int>(i % d8);
    const int tok = it.idx[static_cast<long long>(g) * cap + j];
    const uint8_t* row = (it.src2 && tok >= it.split_row)
                             ? it.src2 + 2 * (g * it.src2_group_stride + static_cast<long long>(tok - it.split_row) * it.src_row_stride)
                             : it.src + 2 * (g * it.src_group_stride + tok * it.src_row_stride);
    const uint4 v = *reinterpret_cast<const uint4*>(row + c * 16);
    *reinterpret_cast<uint4*>(it.dst + 2 * ((static_cast<long long>(g) * cap + j) * d + c * 8)) = v;
  }
}

// dst[g, j, :] = src[g, idx[g, j], :] for j < count[g]  (16-byte chunks; src rows `src_row_stride` elements apart)
__global__ void gather_rows_kernel(const uint8_t* src, long long src_group_stride, long long src_row_stride, const int* idx,
                                   const int* count, int cap, int d, uint8_t* dst) {
  const int g = blockIdx.y, d8 = d / 8;
  const int n = count[g];
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < static_cast<long long>(n) * d8;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i / d8), c = static_cast<int>(i % d8);
    const int tok = idx[static_cast<long long>(g) * cap + j];
    const uint4 v = *reinterpret_cast<const uint4*>(src + 2 * (g * src_group_stride + tok * src_row_stride + c * 8));
    *reinterpret_cast<uint4*>(dst + 2 * ((static_cast<long long>(g) * cap + j) * d + c * 8)) = v;
  }
}

}  // namespace sq
