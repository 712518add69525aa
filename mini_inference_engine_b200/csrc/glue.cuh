// Helpers shared by the memory-bound glue kernels: 8 x bf16 <-> fp32 and the per-128-column e4m3 quantiser.
#pragma once

#include "common.cuh"

namespace mie {

__device__ __forceinline__ void unpack8(const uint4& raw, float (&v)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(p[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 raw;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return raw;
}

__device__ __forceinline__ void unpack4(const uint2& raw, float (&v)[4]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
  const float2 lo = __bfloat1622float2(p[0]), hi = __bfloat1622float2(p[1]);
  v[0] = lo.x, v[1] = lo.y, v[2] = hi.x, v[3] = hi.y;
}
__device__ __forceinline__ uint2 pack4(const float (&v)[4]) {
  uint2 raw;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&raw);
  p[0] = __floats2bfloat162_rn(v[0], v[1]);
  p[1] = __floats2bfloat162_rn(v[2], v[3]);
  return raw;
}

// Eight bf16 values as they come from memory.  A product or a sum of two bf16 values that is rounded to bf16 is one packed
// instruction for two of them (the _rn forms are never contracted): the same bits as fp32 arithmetic and a rounding - exact
// products have 16 bits, and a sum that fp32 would round first has a summand below half a unit of the other.
union Bf16x8 {
  uint4 raw;
  uint32_t word[4];
  __nv_bfloat162 pair[4];
};
// bf16(v * f) of eight values.
__device__ __forceinline__ void scale8(const float (&v)[8], float f, Bf16x8& out) {
#pragma unroll
  for (int i = 0; i < 4; ++i) out.pair[i] = __floats2bfloat162_rn(v[2 * i] * f, v[2 * i + 1] * f);
}

// Launch shape of a kernel that has `lanes` threads for a row: blocks of a part of a wide row, or of several narrow ones
// (block y), as many as leave two blocks per SM.  One row a block: 10000 x 256 through gelu 10.8 us, now 2.9; 16384 x 128
// through SiLU 17.4, now 3.7.
struct RowBlocks {
  int per_row, x, y;
  long long blocks;
  RowBlocks(int rows, int lanes) {
    const int most = rows <= sm_count() ? 128 : 512;  // few rows: more, smaller blocks
    per_row = (lanes + most - 1) / most;
    x = per_row > 1 ? ((lanes + per_row - 1) / per_row + 31) / 32 * 32 : lanes;
    const int room = 256 / x, enough = rows / (2 * sm_count());
    y = room < enough ? room : enough;
    if (per_row > 1 || y < 1) y = 1;
    blocks = (long long)((rows + y - 1) / y) * per_row;
  }
  dim3 grid() const { return dim3((unsigned)blocks); }
  dim3 block() const { return dim3((unsigned)x, (unsigned)y); }
};

// a / b from y, an approximation of 1 / b: quotient, its exact remainder, correction.  Correctly rounded when y is the
// correctly rounded reciprocal (Markstein's theorem), else but for quotients within 2^-20 units of a tie.  Three
// instructions where an IEEE division takes about ten.  a, b and y must be finite.
__device__ __forceinline__ float corrected_quotient(float a, float b, float y) {
  const float q = a * y;
  return fmaf(-fmaf(q, b, -a), y, q);  // signs placed so that a zero keeps its own
}

// g / (1 + exp(-slope g)).
__device__ __forceinline__ float gate_sigmoid(float g, float slope = 1.f) { return g / (1.f + expf(-slope * g)); }

// The same for a result that is rounded to 16 bits: a corrected quotient.
__device__ __forceinline__ float gate_sigmoid16(float g, float slope) {
  const float d = 1.f + expf(-slope * g);
  // a reciprocal near or below the smallest normal number, an infinite gate
  if (d > 1e37f || fabsf(g) > 3.4e38f) return __fdiv_rn(g, d);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return corrected_quotient(g, d, y);
}

// g / (1 + 2^e) from the approximate exponential and reciprocal, each within about 2^-22; a relative error of e carries over
// as |e| ln 2 times as much.  The reciprocal of a denominator above kGateLimit is flushed to zero.
constexpr float kGateLimit = 5e37f, kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float gate_denominator(float e) {
  float t;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(e));
  return 1.f + t;
}
__device__ __forceinline__ float gate_quotient(float g, float denominator) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(denominator));
  return g * y;
}
// SiLU of a bf16 value, to be rounded to bf16: every one of the 65,536 comes out as the division's result does, though before
// the rounding the error grows with the gate, 2^-17 at -88.
__device__ __forceinline__ float silu16(float g) {
  const float d = gate_denominator(g * -kLog2e);
  return d > kGateLimit ? gate_sigmoid(g) : gate_quotient(g, d);
}
// Eight of them with one test for all.
__device__ __forceinline__ void silu8(const float (&g)[8], float (&f)[8]) {
  float top = 0.f;  // NaN passes the test and comes through the quotient
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[j] = gate_denominator(g[j] * -kLog2e);
    top = fmaxf(top, f[j]);
  }
  const bool plain = top <= kGateLimit;
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = plain ? gate_quotient(g[j], f[j]) : gate_sigmoid(g[j]);
}

// v[0..n) / denom as e4m3, two values per 16 bits.  denom >= 1e-12; quotients that e4m3 does not round to zero are exact
// IEEE quotients.
template <int N>
__device__ __forceinline__ void quantize_values(const float (&v)[N], float denom, uint32_t (&packed)[N / 4]) {
  float q[N];
  if (denom < 1e38f) {
    const float y = __frcp_rn(denom);
#pragma unroll
    for (int j = 0; j < N; ++j) q[j] = corrected_quotient(v[j], denom, y);
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) q[j] = __fdiv_rn(v[j], denom);
  }
#pragma unroll
  for (int h = 0; h < N / 4; ++h) {
    const __nv_fp8x2_storage_t lo =
        __nv_cvt_float2_to_fp8x2(make_float2(q[4 * h], q[4 * h + 1]), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi =
        __nv_cvt_float2_to_fp8x2(make_float2(q[4 * h + 2], q[4 * h + 3]), __NV_SATFINITE, __NV_E4M3);
    packed[h] = (uint32_t)lo | ((uint32_t)hi << 16);
  }
}

// Quantise 8 values held by each of 16 consecutive lanes (one 128-column group): this lane's eight e4m3
// bytes and the group's raw scale (amax / 448).
__device__ __forceinline__ void quantize_group(const float (&v)[8], uint32_t (&packed)[2], float& scale) {
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  scale = __fdiv_rn(amax, 448.0f);
  quantize_values(v, fmaxf(scale, 1e-12f), packed);
}
__device__ __forceinline__ void quantize_group_store(const float (&v)[8], uint8_t* q_dst, float* scale_dst,
                                                     bool scale_writer) {
  uint32_t packed[2];
  float scale;
  quantize_group(v, packed, scale);
  if (q_dst != nullptr) *reinterpret_cast<uint2*>(q_dst) = make_uint2(packed[0], packed[1]);
  if (scale_writer && scale_dst != nullptr) *scale_dst = scale;
}

}  // namespace mie
