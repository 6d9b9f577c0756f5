// Elementwise / row-reduction kernels around the attention kernels: q pre-scaling, bf16->f16 copy of V,
// K-mean centring and the fake quantisers of the adapter (sqattn/attn_replacer.py:334-365,
// sqattn/fake_quant.py).  All of them are HBM-bound streaming passes with 16-byte accesses.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "ptx.cuh"

namespace sq {

constexpr float kLog2e = 1.44269504f;  // the literal the reference launchers use

template <bool BF16>
__device__ __forceinline__ float to_f32(uint16_t v) {
  if (BF16) return __uint_as_float(static_cast<uint32_t>(v) << 16);
  return __half2float(__ushort_as_half(v));
}
template <bool BF16>
__device__ __forceinline__ uint16_t from_f32(float f) {
  if (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(f));
  return __half_as_ushort(__float2half_rn(f));
}
template <bool BF16>
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = to_f32<BF16>(static_cast<uint16_t>(w[i] & 0xffffu));
    f[2 * i + 1] = to_f32<BF16>(static_cast<uint16_t>(w[i] >> 16));
  }
}
template <bool BF16>
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    w[i] = static_cast<uint32_t>(from_f32<BF16>(f[2 * i])) | (static_cast<uint32_t>(from_f32<BF16>(f[2 * i + 1])) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// A 16-bit float as an fp64 whose exponent field is the narrow type's: the value is off by the power of two
// kNarrowScale, which the fused multiply-add below puts right exactly (zeros and subnormals come out right as well).
// An integer shift and one DFMA instead of a conversion to fp64, which runs at a quarter of the fp64 rate.
template <bool BF16>
__device__ __forceinline__ double narrow_as_double(uint32_t h) {
  return __hiloint2double(static_cast<int>(((h & 0x7fffu) << (BF16 ? 13 : 10)) | ((h & 0x8000u) << 16)), 0);
}
template <bool BF16>
__device__ __forceinline__ double narrow_scale() { return __hiloint2double(((BF16 ? 896 : 1008) + 1023) << 20, 0); }
// an infinity or a NaN among two 16-bit values: they have no exponent of their own in the shifted form
template <bool BF16>
__device__ __forceinline__ bool narrow_special(uint32_t w) {
  constexpr uint32_t kExp = BF16 ? 0x7f807f80u : 0x7c007c00u, kOne = BF16 ? 0x00800080u : 0x04000400u;
  return (((w & kExp) + kOne) & 0x80008000u) != 0u;
}

struct View4 {  // [B,H,N,D] through element strides
  const uint8_t* ptr;
  long long sb, sh, sn;
  int b, h, n, d;
};
struct OutStrides {  // element strides of an output [B,H,N,D] (contiguous HND or token-major NHD)
  long long sb, sh, sn;
};

// out (contiguous [B,H,N,D]) = f(in): kOp 0: x * scale rounded to the input dtype (q pre-scaling,
// attn_triton_mix_relative.py:383-385); kOp 1: bf16 -> f16 (the kernel-side v.to(fp16), attn_triton.py:84).
template <bool BF16, int kOp>
__global__ void __launch_bounds__(256) strided_map_kernel(View4 in, uint8_t* out, float scale) {
  // a (batch, head) per blockIdx.y: no division but the shift by d / 8 in a thread's loop
  const int shift = in.d == 128 ? 4 : 3;
  const long long per = static_cast<long long>(in.n) << shift;
  for (int bh = blockIdx.y; bh < in.b * in.h; bh += gridDim.y) {
    const uint8_t* src = in.ptr + 2 * (bh / in.h * in.sb + bh % in.h * in.sh);
    uint8_t* dst = out + bh * per * 16;
    for (long long idx = blockIdx.x * 256ll + threadIdx.x; idx < per; idx += gridDim.x * 256ll) {
      const int c = static_cast<int>(idx) & ((1 << shift) - 1);
      const uint4 v = *reinterpret_cast<const uint4*>(src + 2 * ((idx >> shift) * in.sn + c * 8));
      float f[8];
      unpack8<BF16>(v, f);
      uint4 o;
      if (kOp == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] *= scale;
        o = pack8<BF16>(f);
      } else {
        o = pack8<false>(f);
      }
      *reinterpret_cast<uint4*>(dst + idx * 16) = o;
    }
  }
}

// ---- K mean over the sequence, deterministic two-phase reduction -------------------------------------
constexpr int kMeanChunks = 64;

// partial[bh][chunk][d] = sum over the chunk's rows of k[b, n, h, d]; red: [256 / (d / 8)][d] fp32 of shared memory
template <bool BF16>
__device__ __forceinline__ void kmean_partial_body(const View4& k, float* partial, int bh, int chunk, float* red) {
  const int b = bh / k.h, h = bh % k.h;
  const int d8 = k.d / 8, lanes = blockDim.x / d8;
  const int c = threadIdx.x % d8, rl = threadIdx.x / d8;
  const int rows_per = (k.n + kMeanChunks - 1) / kMeanChunks;
  const int r0 = chunk * rows_per, r1 = min(k.n, r0 + rows_per);
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (rl < lanes) {
    for (int n = r0 + rl; n < r1; n += lanes) {
      const uint4 v = *reinterpret_cast<const uint4*>(k.ptr + 2 * (b * k.sb + h * k.sh + n * k.sn + c * 8));
      float f[8];
      unpack8<BF16>(v, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
    }
  }
  if (rl < lanes) {
#pragma unroll
    for (int i = 0; i < 8; ++i) red[rl * k.d + c * 8 + i] = acc[i];
  }
  __syncthreads();
  if (threadIdx.x < k.d) {
    float s = 0.f;
    for (int j = 0; j < lanes; ++j) s += red[j * k.d + threadIdx.x];
    partial[(static_cast<long long>(bh) * kMeanChunks + chunk) * k.d + threadIdx.x] = s;
  }
}
template <bool BF16>
__global__ void kmean_partial_kernel(View4 k, float* partial) {
  extern __shared__ float red[];
  kmean_partial_body<BF16>(k, partial, blockIdx.y, blockIdx.x, red);
}
// sums[bh][d] = the partials in chunk order (the sequence-parallel path all-reduces the sums of the shards)
__global__ void kmean_final_kernel(const float* partial, float* sums, int d) {
  const int bh = blockIdx.x;
  if (threadIdx.x < d) {
    float s = 0.f;
    for (int c = 0; c < kMeanChunks; ++c) s += partial[(static_cast<long long>(bh) * kMeanChunks + c) * d + threadIdx.x];
    sums[bh * d + threadIdx.x] = s;
  }
}

// ---- fake quantisers ---------------------------------------------------------------------------------
__device__ __forceinline__ float round_mode(float x, int half_even) { return half_even ? rintf(x) : roundf(x); }

// float_quantize of the reference (fake_quant.py:151-204) with its quirks: no subnormals, the mantissa
// never carries into the next binade, exponent clipped to 2^(e-1)-1.
__device__ __forceinline__ float float_quantize_dev(float x, int e_bits, int m_bits, int half_even) {
  const int bias = (1 << (e_bits - 1)) - 1;
  const float eps = exp2f(-static_cast<float>(m_bits));
  const float max_exp = static_cast<float>((1 << (e_bits - 1)) - 1);
  const float min_exp = static_cast<float>(1 - bias);
  const float sign = (x > 0.f) ? 1.f : ((x < 0.f) ? -1.f : 0.f);
  const float a = fabsf(x);
  if (a == 0.f) return 0.f;
  const float ex = floorf(log2f(a + 1e-30f));
  const float frac = __fdiv_rn(a, exp2f(ex)) - 1.0f;
  const float exc = fminf(fmaxf(ex, min_exp), max_exp);
  float fq = round_mode(__fdiv_rn(frac, eps), half_even) * eps;
  fq = fminf(fmaxf(fq, 0.0f), 1.0f - eps);
  float xq = (1.0f + fq) * exp2f(exc) * sign;
  const float max_val = (2.0f - eps) * exp2f(max_exp);
  return fminf(fmaxf(xq, -max_val), max_val);
}

// quant -> dequant of one value on the integer grid of `scale`, with the reference's divisions
__device__ __forceinline__ float int_grid_value(float x, float scale, float qmax, int half_even) {
  float q = round_mode(__fdiv_rn(x, scale), half_even);
  q = fminf(fmaxf(q, -qmax - 1.0f), qmax);
  return q * scale;
}

// quant -> dequant of one value given the row's absmax (clipped at 1e-5).
//   qtype 0: integer grid with `qmax` (127 / 7), clamp to [-qmax-1, qmax]  (fake_quant.py:114-125)
//   qtype 1/2: emulated e4m3 / e5m2                                         (fake_quant.py:231-248)
__device__ __forceinline__ float fake_quant_value(float x, float absmax, int qtype, float qmax, int half_even) {
  if (qtype == SQATTN_QTYPE_INT) return int_grid_value(x, __fdiv_rn(absmax, qmax), qmax, half_even);
  const float fmax = (qtype == SQATTN_QTYPE_E4M3) ? 448.0f : 57344.0f;
  const float scale = __fdiv_rn(absmax, fmax);
  float s = fminf(fmaxf(__fdiv_rn(x, scale), -fmax), fmax);
  s = float_quantize_dev(s, qtype == SQATTN_QTYPE_E4M3 ? 4 : 5, qtype == SQATTN_QTYPE_E4M3 ? 3 : 2, half_even);
  return s * scale;
}

// The nearest integers of two values below 2^22 in magnitude: adding and taking off 1.5 * 2^23 leaves them (ties to even; a
// negative zero comes out positive).  The conversion unit's own rounding runs at an eighth of this rate.
__device__ __forceinline__ uint64_t rint2_small(uint64_t x2) {
  const uint64_t m = f32x2_pack(12582912.0f, 12582912.0f);
  return f32x2_sub(f32x2_add(x2, m), m);
}
template <bool BF16>
__device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi) {
  lo = to_f32<BF16>(static_cast<uint16_t>(w & 0xffffu));
  hi = BF16 ? __uint_as_float(w & 0xffff0000u) : to_f32<BF16>(static_cast<uint16_t>(w >> 16));
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) { return BF16 ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi); }
// largest magnitude of 8 values, in their own type (a NaN counts as nothing beside a number)
template <bool BF16>
__device__ __forceinline__ float absmax8(const uint4& x) {
  auto larger = [](uint32_t a, uint32_t b) {
    uint32_t r;
    if (BF16) asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  };
  constexpr uint32_t kAbs = 0x7fff7fffu;
  float lo, hi;
  unpack2<BF16>(larger(larger(x.x & kAbs, x.y & kAbs), larger(x.z & kAbs, x.w & kAbs)), lo, hi);
  return fmaxf(lo, hi);
}

// The integer grid for 8 values of one row, on packed fp32 pairs, returning the 8 results
// rounded to the 16-bit type (and, for queries, multiplied by q_scale and rounded again) as four packed words.
// q = x * inv, inv = 1/scale, is within 2e-5 of the exact quotient x / scale (|q| <= qmax * (1 + 2^-22), so the clamp of the
// reference never acts), hence unless q lies within 1e-4 of a half-integer its nearest integer IS round(x / scale) in
// either rounding mode; a group with such a value (rare) is redone with exact divisions.  The bits are those of
// fake_quant_value(..., INT, ...).  A result has the sign of its input, zeros too: the sign bits are put back two at a time.
template <bool BF16, bool kScale>
__device__ __forceinline__ uint4 fake_quant_int_row8(const uint4& x, float scale, float inv, float qmax, int half_even, float q_scale) {
  const uint64_t inv2 = f32x2_pack(inv, inv), sc2 = f32x2_pack(scale, scale), qs2 = f32x2_pack(q_scale, q_scale);
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
  float g[8];
  float worst = 0.f;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float a, b, d0, d1;
    unpack2<BF16>(w[p], a, b);
    const uint64_t q2 = f32x2_mul(f32x2_pack(a, b), inv2);
    const uint64_t r2 = rint2_small(q2);
    f32x2_unpack(f32x2_sub(q2, r2), d0, d1);
    worst = max3(worst, fabsf(d0), fabsf(d1));
    f32x2_unpack(f32x2_mul(r2, sc2), g[2 * p], g[2 * p + 1]);
  }
  if (worst > 0.4999f) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float a, b;
      unpack2<BF16>(w[p], a, b);
      g[2 * p] = int_grid_value(a, scale, qmax, half_even);
      g[2 * p + 1] = int_grid_value(b, scale, qmax, half_even);
    }
  }
  uint32_t out[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t v = pack2<BF16>(g[2 * p], g[2 * p + 1]);
    if (kScale) {
      float a, b;
      unpack2<BF16>(v, a, b);
      f32x2_unpack(f32x2_mul(f32x2_pack(a, b), qs2), a, b);
      v = pack2<BF16>(a, b);
    }
    out[p] = v | (w[p] & 0x80008000u);
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}

// "per_channel" fake-quant of V for the 4 channels c of token n: one range per (token, channel), taken over batch and
// heads (fake_quant.py:30-32 with a [B,H,N,D] tensor).  Output in f16.  Four channels a thread (8-byte accesses): with
// eight, the ranges, scales and held values of a thread left two blocks per SM and the pass took twice as long.
template <bool BF16, bool kInt>
__device__ __forceinline__ void quant_v_body(const View4& v, uint8_t* out, const OutStrides& os, int qtype, int half_even, int n, int c) {
  constexpr int kHeld = 4;   // (batch, head) pairs kept in registers: their loads are in flight together
  const int bh = v.b * v.h;
  struct Walk {              // byte offsets of the pairs in turn
    long long in, out;
    int h;
  };
  auto next = [&](Walk& w) {
    w.in += 2 * v.sh; w.out += 2 * os.sh;
    if (++w.h == v.h) { w.h = 0; w.in += 2 * (v.sb - v.h * v.sh); w.out += 2 * (os.sb - v.h * os.sh); }
  };
  auto unpack4 = [](const uint2& r, float (&f)[4]) {
    f[0] = to_f32<BF16>(static_cast<uint16_t>(r.x & 0xffffu)); f[1] = to_f32<BF16>(static_cast<uint16_t>(r.x >> 16));
    f[2] = to_f32<BF16>(static_cast<uint16_t>(r.y & 0xffffu)); f[3] = to_f32<BF16>(static_cast<uint16_t>(r.y >> 16));
  };
  const Walk start{2 * (n * v.sn + c * 4), 2 * (n * os.sn + c * 4), 0};
  float amax[4] = {0, 0, 0, 0};
  uint2 raw[kHeld];
  Walk w = start;
#pragma unroll
  for (int u = 0; u < kHeld; ++u, next(w)) raw[u] = u < bh ? *reinterpret_cast<const uint2*>(v.ptr + w.in) : make_uint2(0u, 0u);
  auto widen = [&](const uint2& r) {
    float f[4];
    unpack4(r, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) amax[i] = fmaxf(amax[i], fabsf(f[i]));
  };
#pragma unroll
  for (int u = 0; u < kHeld; ++u) widen(raw[u]);
#pragma unroll 4
  for (int u = kHeld; u < bh; ++u, next(w)) widen(*reinterpret_cast<const uint2*>(v.ptr + w.in));
  float scale[4], inv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    amax[i] = fmaxf(amax[i], 1e-5f);
    scale[i] = __fdiv_rn(amax[i], 127.0f);
    inv[i] = __fdiv_rn(1.0f, scale[i]);
  }
  auto store = [&](const uint2& r, long long off) {
    float f[4], g[4];
    unpack4(r, f);
    bool sure = kInt;
    if (kInt) {   // the reciprocal and its check: see fake_quant_int_row8; a NaN is never sure, the clamp decides about it
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float q = f[i] * inv[i], rq = rintf(q);
        sure = sure && fabsf(q - rq) <= 0.4999f;
        g[i] = rq * scale[i];
      }
    }
    if (!sure) {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = fake_quant_value(f[i], amax[i], qtype, 127.0f, half_even);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) g[i] = to_f32<BF16>(from_f32<BF16>(g[i]));
    *reinterpret_cast<uint2*>(out + off) = make_uint2(pack_f16x2(g[0], g[1]), pack_f16x2(g[2], g[3]));
  };
  w = start;
#pragma unroll
  for (int u = 0; u < kHeld; ++u, next(w))
    if (u < bh) store(raw[u], w.out);
#pragma unroll 1
  for (int u = kHeld; u < bh; ++u, next(w)) store(*reinterpret_cast<const uint2*>(v.ptr + w.in), w.out);
}

// Preparation, first launch: column sums of K (blocks [0, sum_blocks): kMeanChunks per (batch, head)) and all of V.
template <bool BF16, bool kInt>
__global__ void __launch_bounds__(256, 4)
prep_sums_v_kernel(View4 k, float* partial, int sum_blocks, View4 v, uint8_t* out_v, OutStrides os, int qtype, int half_even) {
  __shared__ float red[256 * 8];
  griddep_launch();   // the second launch's query blocks need nothing from here
  if (static_cast<int>(blockIdx.x) < sum_blocks) {
    kmean_partial_body<BF16>(k, partial, blockIdx.x / kMeanChunks, blockIdx.x % kMeanChunks, red);
    return;
  }
  const int d4 = v.d / 4;
  const long long total = static_cast<long long>(v.n) * d4;
  for (long long idx = (blockIdx.x - sum_blocks) * 256ll + threadIdx.x; idx < total; idx += (gridDim.x - sum_blocks) * 256ll)
    quant_v_body<BF16, kInt>(v, out_v, os, qtype, half_even, static_cast<int>(idx / d4), static_cast<int>(idx % d4));
}

// Per-token fake-quant of block `blk` of the rows of one (batch, head) of Q or K.
// kIsK: subtract the (dtype-rounded) sequence mean first, no scaling of the result.
// Q: results are multiplied by 1/sqrt(D)*log2e in the input dtype.
// One 16-lane group per row (D = 128) or one 8-lane group (D = 64); 16-byte loads and stores.
constexpr int kQuantRowsPerThread = 4;   // rows in flight per lane group: four independent 16-byte loads per thread
struct QuantRows {
  View4 x;
  uint8_t *out8, *out4;
  OutStrides os;
  int blocks;   // per (batch, head)
};
template <bool BF16, bool kIsK, bool kInt>
__device__ __forceinline__ void quant_rows_body(const QuantRows& r, const float* mean, int bh, int blk, int qtype, int half_even, float q_scale) {
  constexpr int kUnroll = kQuantRowsPerThread;
  const View4& x = r.x;
  const int d8 = x.d / 8;
  const int rows_per_block = 256 / d8;
  const int c = threadIdx.x % d8;
  const int b = bh / x.h, h = bh % x.h;
  const uint8_t* in_base = x.ptr + 2 * (b * x.sb + h * x.sh + c * 8);
  const long long out_base = (b * r.os.sb + h * r.os.sh + c * 8) * 2;
  float mvals[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (kIsK) {
#pragma unroll
    for (int i = 0; i < 8; ++i) mvals[i] = to_f32<BF16>(from_f32<BF16>(mean[c * 8 + i]));
  }
  const int n0 = blk * rows_per_block * kUnroll + threadIdx.x / d8;
  uint4 raw[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int n = n0 + u * rows_per_block;
    raw[u] = n < x.n ? *reinterpret_cast<const uint4*>(in_base + 2 * (static_cast<long long>(n) * x.sn)) : make_uint4(0u, 0u, 0u, 0u);
  }
  float amax[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    if (kIsK) {
      float f[8];
      unpack8<BF16>(raw[u], f);
      raw[u] = make_uint4(pack2<BF16>(f[0] - mvals[0], f[1] - mvals[1]), pack2<BF16>(f[2] - mvals[2], f[3] - mvals[3]),
                          pack2<BF16>(f[4] - mvals[4], f[5] - mvals[5]), pack2<BF16>(f[6] - mvals[6], f[7] - mvals[7]));
    }
    amax[u] = absmax8<BF16>(raw[u]);
  }
  // The largest of each row over its lanes, transposed: lane c ends up with row c & 3 and is the one that divides for it.
  static_assert(kUnroll == 4, "two exchange steps");
  {
    const bool b0 = c & 1, b1 = c & 2;
    const float k0 = fmaxf(b0 ? amax[1] : amax[0], __shfl_xor_sync(0xffffffffu, b0 ? amax[0] : amax[1], 1));
    const float k1 = fmaxf(b0 ? amax[3] : amax[2], __shfl_xor_sync(0xffffffffu, b0 ? amax[2] : amax[3], 1));
    amax[0] = fmaxf(b1 ? k1 : k0, __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2));
    for (int o = 4; o < d8; o <<= 1) amax[0] = fmaxf(amax[0], __shfl_xor_sync(0xffffffffu, amax[0], o));
  }
  const float mine = fmaxf(amax[0], 1e-5f);
  const int src = threadIdx.x & 28;   // the lane of the group of four that has row u is src + u
  if (!kInt) {
    // One copy of the emulated format's long code for the four rows, whose registers take turns (28/4 heads, 65536 tokens, e4m3,
    // four copies and one: bf16 1857 and 1433 us, fp16 1834 and 1387; 1000 tokens 41 and 35, 40.5 and 33.5).
#pragma unroll 1
    for (int u = 0; u < kUnroll; ++u) {
      const int n = n0 + u * rows_per_block;
      const float s = __shfl_sync(0xffffffffu, mine, src + u);
      float f[8];
      unpack8<BF16>(raw[0], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        f[e] = to_f32<BF16>(from_f32<BF16>(fake_quant_value(f[e], s, qtype, 127.0f, half_even)));
        if (!kIsK) f[e] *= q_scale;
      }
      if (n < x.n) *reinterpret_cast<uint4*>(r.out8 + out_base + static_cast<long long>(n) * r.os.sn * 2) = pack8<BF16>(f);
      const uint4 first = raw[0];
      raw[0] = raw[1]; raw[1] = raw[2]; raw[2] = raw[3]; raw[3] = first;
    }
  }
  auto rows = [&](uint8_t* out, float qmax) {
    const float scale = __fdiv_rn(mine, qmax), inv = __fdiv_rn(1.0f, scale);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int n = n0 + u * rows_per_block;
      const float s = __shfl_sync(0xffffffffu, scale, src + u), i = __shfl_sync(0xffffffffu, inv, src + u);
      const uint4 v = fake_quant_int_row8<BF16, !kIsK>(raw[u], s, i, qmax, half_even, q_scale);
      if (n < x.n) *reinterpret_cast<uint4*>(out + out_base + static_cast<long long>(n) * r.os.sn * 2) = v;
    }
  };
  if (kInt) rows(r.out8, 127.0f);
  if (r.out4) rows(r.out4, 7.0f);
}

// Preparation, second launch: the rows of Q (first: they do not wait for the first launch) and of K.  K blocks add up the
// column sums of the first launch themselves, in chunk order, unless the caller gave the mean.
// One launch for both, and V beside the sums, instead of five in a row, each of the small ones waiting for its own latency.
// A row's divisions are done by one of its lanes and passed on, its largest magnitude is found in the 16-bit type, and signs go
// back on two at a time: every lane of a row divided for itself before (131072 tokens, queries alone: 540 -> 475 us, 4.0 TB/s).
// Four blocks per SM (64 registers); five (48 registers, 300 bytes spilled) were 1 % slower, three 9 %.
// In a graph, five launches, two, and now, 28/4 heads: 1000 tokens 23.8, 14.8, 13.9 us, 8192 73, 54, 48, 131072 898, 764, 692.
template <bool BF16, bool kInt>
__global__ void __launch_bounds__(256, 4)
prep_rows_kernel(QuantRows q, QuantRows k, int q_blocks, const float* partial, const float* mean, int qtype, int half_even, float q_scale) {
  __shared__ float mean_s[128];
  griddep_launch();
  if (static_cast<int>(blockIdx.x) < q_blocks) {
    quant_rows_body<BF16, false, kInt>(q, nullptr, blockIdx.x / q.blocks, blockIdx.x % q.blocks, qtype, half_even, q_scale);
    griddep_wait();   // this grid does not end before the first launch has: what follows it depends on both
    return;
  }
  griddep_wait();
  const int bh = (blockIdx.x - q_blocks) / k.blocks, d = k.x.d;
  if (static_cast<int>(threadIdx.x) < d) {
    float s = 0.f;
    if (mean) {
      s = mean[bh * d + threadIdx.x];
    } else {
#pragma unroll 16
      for (int c = 0; c < kMeanChunks; ++c) s += partial[(static_cast<long long>(bh) * kMeanChunks + c) * d + threadIdx.x];
      s /= static_cast<float>(k.x.n);
    }
    mean_s[threadIdx.x] = s;
  }
  __syncthreads();
  quant_rows_body<BF16, true, kInt>(k, mean_s, bh, (blockIdx.x - q_blocks) % k.blocks, qtype, half_even, 1.0f);
}

}  // namespace sq
