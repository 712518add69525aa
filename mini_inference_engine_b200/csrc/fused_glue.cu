// Memory-bound glue between the projections: RMSNorm (plain, per-head strided,
// fused with the residual add), SiLU(gate) * up, rotate-half RoPE, and the
// decode-step fusion of q/k-norm + RoPE + KV-cache write.  Each kernel makes one
// pass over HBM with 16-byte accesses and keeps the bf16 rounding points where
// the unfused PyTorch ops round (fp32 math in between).  The norm and SiLU
// kernels can also emit the e4m3 activation + per-128 scales that the next FP8
// GEMM consumes, which removes the separate quantiser pass.
#include "common.cuh"
#include "glue.cuh"
#include "qkv_rows.cuh"

namespace mie {
namespace {

// ---------------------------------------------------------------------------
// Row RMSNorm: a CTA per row, eight columns a thread, cols a multiple of 8 (<= 8 * 1024).  With many rows a CTA goes from
// row to row and requests the next one before it reduces this one; the weight is read once.  Bound by HBM (2 bytes a value
// and tensor, 1 for e4m3), if the arithmetic is packed: 12032 x 2560 with residual, sum and e4m3
// 54.3 us with a CTA per row, now 46.5; 560 rows 5.9 and 4.1, one row 2.9 and 2.1.  (Three CTAs of 320 threads per SM; four
// 50.3, five 55.0; a warp per row 69.)  Narrow rows take as many CTAs as the registers of an SM allow: 12032 x 1024 19.8 us
// with a CTA per row, 25.2 with four per SM, now 17.4.
// ---------------------------------------------------------------------------
struct RowNormParams {
  const __nv_bfloat16* x;
  long long ldx;
  const __nv_bfloat16* residual;  // optional, contiguous rows of `cols`
  __nv_bfloat16* summed;          // optional: x + residual
  const __nv_bfloat16* weight;
  __nv_bfloat16* out;             // optional when only the quantised form is wanted
  uint8_t* q;                     // optional e4m3 output, row stride ldq
  long long ldq;
  float* scales;                  // [cols / 128][scale_ld]
  int scale_ld;
  int rows, cols;
  float eps;
};

// kThreads: the most of the instantiation; kCtas: how many of them an SM holds, all of which go from row to row.
template <int kThreads, int kCtas>
__global__ void __launch_bounds__(kThreads, kCtas) row_norm_kernel(RowNormParams p) {
  __shared__ float red[2][32];
  chain_release();
  chain_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = (blockDim.x + 31) >> 5;
  const int c0 = tid * 8;
  const bool active = c0 < p.cols;
  Bf16x8 x, r, w;
  x.raw = r.raw = w.raw = make_uint4(0, 0, 0, 0);
  auto load = [&](int row) {
    if (!active || row >= p.rows) return;
    x.raw = *reinterpret_cast<const uint4*>(p.x + (long long)row * p.ldx + c0);
    if (p.residual != nullptr) r.raw = *reinterpret_cast<const uint4*>(p.residual + (long long)row * p.cols + c0);
  };
  load(blockIdx.x);
  if (active) w.raw = *reinterpret_cast<const uint4*>(p.weight + c0);  // fetched with the row, not after the reduction
  int turn = 0;
  for (int row = blockIdx.x; row < p.rows; row += gridDim.x, turn ^= 1) {
    Bf16x8 v;
    v.raw = x.raw;
    if (p.residual != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v.pair[i] = __hadd2_rn(x.pair[i], r.pair[i]);
    }
    load(row + gridDim.x);
    if (active && p.summed != nullptr) *reinterpret_cast<uint4*>(p.summed + (long long)row * p.cols + c0) = v.raw;
    float f[8], ss = 0.f;
    unpack8(v.raw, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    ss = warp_sum(ss);
    if (lane == 0) red[turn][warp] = ss;  // the other half may still be read: the barrier of this row is behind that
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < warps; ++i) total += red[turn][i];
    const float inv = rsqrtf(total / (float)p.cols + p.eps);
    Bf16x8 n;
    scale8(f, inv, n);
#pragma unroll
    for (int i = 0; i < 4; ++i) n.pair[i] = __hmul2_rn(w.pair[i], n.pair[i]);
    if (active && p.out != nullptr) *reinterpret_cast<uint4*>(p.out + (long long)row * p.cols + c0) = n.raw;
    if (p.q != nullptr) {
      // Lanes past the row end (cols is a multiple of 128 here) hold nothing and write nothing.
      unpack8(n.raw, f);
      quantize_group_store(f, active ? p.q + (long long)row * p.ldq + c0 : nullptr,
                           active ? p.scales + (long long)(c0 / 128) * p.scale_ld + row : nullptr, (tid & 15) == 0);
    }
  }
}

// ---------------------------------------------------------------------------
// Head RMSNorm: width 128, 16 lanes per (row, head); rows addressed by strides.
// ---------------------------------------------------------------------------
__global__ void head_norm_kernel(const __nv_bfloat16* x, long long outer_stride, long long head_stride, int heads,
                                 const __nv_bfloat16* weight, __nv_bfloat16* out, long long rows_total, float eps) {
  const long long hw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const int l16 = threadIdx.x & 15;
  const bool live = hw < rows_total;
  const long long r = live ? hw : 0;
  const __nv_bfloat16* src = x + (r / heads) * outer_stride + (r % heads) * head_stride + l16 * 8;
  float v[8];
  unpack8(*reinterpret_cast<const uint4*>(src), v);
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float inv = rsqrtf(ss / 128.f + eps);
  float w8[8];
  unpack8(*reinterpret_cast<const uint4*>(weight + l16 * 8), w8);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = round_bf16(w8[j] * round_bf16(v[j] * inv));
  if (live) *reinterpret_cast<uint4*>(out + r * 128 + l16 * 8) = pack8(v);
}

// ---------------------------------------------------------------------------
// SiLU(gate) * up, optional fused quantisation.  Bound by HBM (5 bytes a result when quantised) only with few instructions
// per value: gates by silu8, the product with `up` a packed bf16 multiplication (the same single rounding), corrected
// quotients for e4m3, no index division, several narrow rows a block.  kParts = 2, for many values in rows of whole groups of
// 128 columns: eight lanes have a group, 8 columns and the 8 that lie 64 further, so that what a group takes once (its
// maximum, its scale and reciprocal) is shared by 16 values of a lane; kParts = 1: sixteen lanes a group, a shorter chain.
// 12032 x 9728: 244 us with IEEE divisions, 158 with corrected quotients and 16 lanes a group, now 127 (4096 rows 56.0 and
// 45.2).
// ---------------------------------------------------------------------------
template <int kParts>
__global__ void __launch_bounds__(512)
    silu_mul_kernel(const __nv_bfloat16* gate, const __nv_bfloat16* up, long long ld_in, __nv_bfloat16* out, uint8_t* q,
                    long long ldq, float* scales, int scale_ld, int rows, int cols, int blocks_per_row) {
  constexpr int kLanes = 16 / kParts;  // of a group
  chain_release();
  chain_wait();
  const int first = blockIdx.x / blocks_per_row;
  const int row = first * blockDim.y + threadIdx.y;
  const int in_row = (blockIdx.x - first * blocks_per_row) * blockDim.x + threadIdx.x;
  if (row >= rows || in_row >= cols / (8 * kParts)) return;  // whole groups, where there are groups
  const int c0 = kParts == 2 ? in_row / 8 * 128 + in_row % 8 * 8 : in_row * 8;
  Bf16x8 v[kParts], u[kParts];
#pragma unroll
  for (int x = 0; x < kParts; ++x) {
    v[x].raw = *reinterpret_cast<const uint4*>(gate + (long long)row * ld_in + c0 + x * 64);
    u[x].raw = *reinterpret_cast<const uint4*>(up + (long long)row * ld_in + c0 + x * 64);
  }
  float f[kParts][8], amax = 0.f;
#pragma unroll
  for (int x = 0; x < kParts; ++x) {
    float g[8];
    unpack8(v[x].raw, g);
    silu8(g, f[x]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[x].pair[i] = __hmul2_rn(__floats2bfloat162_rn(f[x][2 * i], f[x][2 * i + 1]), u[x].pair[i]);
    if (out != nullptr) *reinterpret_cast<uint4*>(out + (long long)row * cols + c0 + x * 64) = v[x].raw;
    unpack8(v[x].raw, f[x]);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(f[x][j]));
  }
  if (q == nullptr) return;
  const int lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31;
  const uint32_t group = ((1u << kLanes) - 1) << (lane & ~(kLanes - 1));
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(group, amax, o));
  const float scale = __fdiv_rn(amax, 448.0f), denom = fmaxf(scale, 1e-12f);
#pragma unroll
  for (int x = 0; x < kParts; ++x) {
    uint32_t packed[2];
    quantize_values(f[x], denom, packed);
    *reinterpret_cast<uint2*>(q + (long long)row * ldq + c0 + x * 64) = make_uint2(packed[0], packed[1]);
  }
  if ((lane & (kLanes - 1)) == 0) scales[(long long)(c0 / 128) * scale_ld + row] = scale;
}

// ---------------------------------------------------------------------------
// RoPE on [B, H, T, D] (D <= 256, even): one warp per (b, h, t) row.
// ---------------------------------------------------------------------------
__global__ void rope_kernel(const __nv_bfloat16* x, long long sb, long long sh, long long st,
                            const __nv_bfloat16* cos, const __nv_bfloat16* sin, long long cs_b, long long cs_t,
                            __nv_bfloat16* out, long long ob, long long oh, long long ot, int heads, int seq,
                            int dim, long long rows_total) {
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= rows_total) return;
  const int t = (int)(warp % seq), h = (int)((warp / seq) % heads);
  const long long b = warp / ((long long)seq * heads);
  const __nv_bfloat16* src = x + b * sb + h * sh + t * st;
  const __nv_bfloat16* c = cos + b * cs_b + t * cs_t;
  const __nv_bfloat16* s = sin + b * cs_b + t * cs_t;
  __nv_bfloat16* dst = out + b * ob + h * oh + t * ot;
  const int half = dim / 2;
  for (int i = lane; i < half; i += 32) {
    const float x1 = __bfloat162float(src[i]), x2 = __bfloat162float(src[i + half]);
    const float o1 = round_bf16(x1 * __bfloat162float(c[i])) + round_bf16(-x2 * __bfloat162float(s[i]));
    const float o2 =
        round_bf16(x2 * __bfloat162float(c[i + half])) + round_bf16(x1 * __bfloat162float(s[i + half]));
    dst[i] = __float2bfloat16_rn(o1);
    dst[i + half] = __float2bfloat16_rn(o2);
  }
}

// ---------------------------------------------------------------------------
// q/k RMSNorm + RoPE + KV-cache write over a merged qkv row (head_dim 128).  A block per token (or several), 16 lanes per head, eight
// consecutive dims a lane (partner dims d +/- 64 sit 8 lanes away): a lane's cos / sin entries, position and page serve
// all the heads of its half-warp, whose rows are in flight together.  A warp per (token, head) with 8-byte accesses
// looked all of that up per head: 12032 tokens of 48 heads 185 us; fp32 arithmetic with a rounding after each operation 137,
// packed bf16 90 (147 MB in, 147 MB out; 4096 tokens 49 and 33).
// ---------------------------------------------------------------------------
// Eight bf16 values, 16-byte aligned when `wide`, else 8-byte.
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p, bool wide) {
  if (wide) return *reinterpret_cast<const uint4*>(p);
  const uint2 lo = *reinterpret_cast<const uint2*>(p), hi = *reinterpret_cast<const uint2*>(p + 4);
  return make_uint4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const uint4& v, bool wide) {
  if (wide) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
    *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
  }
}

constexpr int kQkvBatch = 3;  // head rows of a half-warp in flight

__global__ void __launch_bounds__(256) qkv_post_kernel(QkvParams p) {
  chain_release();
  chain_wait();
  const int t = blockIdx.x, l16 = threadIdx.x & 15;
  const int heads_total = p.q_heads + 2 * p.kv_heads, half_warps = (blockDim.x >> 4) * gridDim.y;
  const __nv_bfloat16* src = p.qkv + (long long)t * p.ld + l16 * 8;
  const int h_first = blockIdx.y * (blockDim.x >> 4) + (threadIdx.x >> 4);
  uint4 raw[kQkvBatch];
  auto load_batch = [&](int h0) {
#pragma unroll
    for (int u = 0; u < kQkvBatch; ++u) {
      const int h = h0 + u * half_warps;
      if (h >= heads_total)
        raw[u] = make_uint4(0, 0, 0, 0);
      else
        raw[u] = load8(src + h * 128, p.wide);
    }
  };
  load_batch(h_first);
  long long pos, page;
  qkv_place(p, t, threadIdx.x == 0 && blockIdx.y == 0, pos, page);
  const long long cpos = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
  const __nv_bfloat16* cs = p.cos_sin + cpos * 256 + l16 * 8;
  Bf16x8 c, s;  // rotate_half is (-x2, x1): the sign goes to the sines of the lower half
  c.raw = load8(cs, p.wide);
  s.raw = load8(cs + 128, p.wide);
#pragma unroll
  for (int i = 0; i < 4; ++i) s.word[i] ^= l16 < 8 ? 0x80008000u : 0u;
  const int slot = (int)((pos < 0 ? 0 : pos) % p.block_size);

  for (int h0 = h_first; h0 - h_first < heads_total; h0 += kQkvBatch * half_warps) {
    if (h0 != h_first) load_batch(h0);
#pragma unroll
    for (int u = 0; u < kQkvBatch; ++u) {
      const int h = h0 + u * half_warps;  // a half-warp past the last head stays for the shuffles
      if (h - h_first >= heads_total) break;
      const bool is_q = h < p.q_heads, is_v = h >= p.q_heads + p.kv_heads, live = h < heads_total;
      float v[8];
      unpack8(raw[u], v);
      const float inv = rsqrtf(half_warp_square_sum(v, l16) / 128.f + p.eps);
      Bf16x8 w, n, o;
      w.raw = load8((is_q ? p.q_weight : p.k_weight) + l16 * 8, p.wide);
      scale8(v, inv, n);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        n.pair[i] = __hmul2_rn(w.pair[i], n.pair[i]);
        Bf16x8 partner;
        partner.word[0] = __shfl_xor_sync(0xffffffffu, n.word[i], 8);
        o.pair[i] = __hadd2_rn(__hmul2_rn(n.pair[i], c.pair[i]), __hmul2_rn(partner.pair[0], s.pair[i]));
      }
      const uint4 result = is_v ? raw[u] : o.raw;
      // e4m3 pool: one scale per (token, KV head), amax of the 128 bf16 values / 448, the row divided by it and rounded
      // to e4m3 (the activation quantiser's rule).  Every half-warp takes part, whatever its head is.
      uint32_t packed[2];
      float scale;
      if (p.kv8_pool != nullptr) {
        float f[8];
        unpack8(result, f);
        quantize_group(f, packed, scale);
      }
      if (is_q) {
        store8(p.q_out + ((long long)t * p.q_heads + h) * 128 + l16 * 8, result, p.wide);
        continue;
      }
      if (!live || page < 0) continue;
      const int kvh = is_v ? h - p.q_heads - p.kv_heads : h - p.q_heads;
      if (p.kv8_pool != nullptr) {
        uint8_t* row = p.kv8_pool + page * p.kv8_page_stride + ((long long)kvh * 2 + (is_v ? 1 : 0)) * 2048 + slot * 128;
        if (p.wide) {
          *reinterpret_cast<uint2*>(row + l16 * 8) = make_uint2(packed[0], packed[1]);
        } else {
          *reinterpret_cast<uint32_t*>(row + l16 * 8) = packed[0];
          *reinterpret_cast<uint32_t*>(row + l16 * 8 + 4) = packed[1];
        }
        if (l16 == 0) p.kv8_scales[((page * p.kv_heads + kvh) * 2 + (is_v ? 1 : 0)) * 16 + slot] = scale;
        continue;
      }
      const long long* st = is_v ? p.vb_s : p.kb_s;
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(is_v ? p.value_blocks : p.key_blocks) + page * st[0] +
                           (long long)kvh * st[1] + slot * st[2] + l16 * 8;
      store8(dst, result, p.wide);
    }
  }
}

}  // namespace
}  // namespace mie

using namespace mie;

extern "C" int mie_rms_norm(const void* x, int64_t ldx, const void* residual, void* summed, const void* weight,
                            void* out, void* q, int64_t ldq, float* scales, int32_t scale_ld, int32_t rows,
                            int32_t cols, float eps, void* stream) {
  MIE_CHECK_ARG(x && weight && (out || q), "null pointer");
  MIE_CHECK_ARG(rows >= 0 && cols >= 8 && cols % 8 == 0 && cols <= 8192, "cols must be a multiple of 8 in [8, 8192]");
  MIE_CHECK_ARG(ldx % 8 == 0 && aligned16(x) && aligned16(weight) && (!out || aligned16(out)) &&
                    (!residual || aligned16(residual)) && (!summed || aligned16(summed)),
                "rows must be 16-byte aligned");
  MIE_CHECK_ARG(!q || (scales && cols % 128 == 0 && scale_ld >= rows && ldq >= cols && ldq % 8 == 0),
                "fused quantisation needs cols %% 128 == 0 and scale storage");
  if (rows == 0) return MIE_OK;
  RowNormParams p{(const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)residual, (__nv_bfloat16*)summed,
                  (const __nv_bfloat16*)weight, (__nv_bfloat16*)out, (uint8_t*)q, ldq, scales, scale_ld, rows, cols,
                  eps};
  const int threads = ((cols / 8) + 31) / 32 * 32;
  const auto launch = [&](auto kernel, int per_sm) {
    const int ctas = sm_count() * per_sm;
    return launch_chained(kernel, dim3(rows < ctas ? rows : ctas), dim3(threads), 0, (cudaStream_t)stream, p);
  };
  // 56 registers a thread, of 64 Ki an SM.
  MIE_CUDA(threads <= 256   ? launch(row_norm_kernel<256, 4>, 1152 / threads)
           : threads <= 384 ? launch(row_norm_kernel<384, 3>, 3)
           : threads <= 512 ? launch(row_norm_kernel<512, 2>, 2)
                            : launch(row_norm_kernel<1024, 1>, 1));
  MIE_LAUNCH_CHECK("row_norm_kernel");
  return MIE_OK;
}

extern "C" int mie_head_rms_norm(const void* x, int64_t outer_stride, int64_t head_stride, int32_t heads,
                                 const void* weight, void* out, int64_t rows_total, float eps, void* stream) {
  MIE_CHECK_ARG(x && weight && out && heads >= 1 && rows_total >= 0, "invalid head-norm arguments");
  MIE_CHECK_ARG(outer_stride % 8 == 0 && head_stride % 8 == 0 && aligned16(x) && aligned16(weight) && aligned16(out),
                "head rows must be 16-byte aligned");
  if (rows_total == 0) return MIE_OK;
  const int threads = 256;
  const long long blocks = (rows_total * 16 + threads - 1) / threads;
  head_norm_kernel<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, outer_stride, head_stride, heads, (const __nv_bfloat16*)weight, (__nv_bfloat16*)out,
      rows_total, eps);
  MIE_LAUNCH_CHECK("head_norm_kernel");
  return MIE_OK;
}

extern "C" int mie_silu_mul(const void* gate, const void* up, int64_t ld_in, void* out, void* q, int64_t ldq,
                            float* scales, int32_t scale_ld, int32_t rows, int32_t cols, void* stream) {
  MIE_CHECK_ARG(gate && up && (out || q), "null pointer");
  MIE_CHECK_ARG(rows >= 0 && cols >= 8 && cols % 8 == 0 && ld_in % 8 == 0, "cols and row stride must be multiples of 8");
  MIE_CHECK_ARG(aligned16(gate) && aligned16(up) && (!out || aligned16(out)), "rows must be 16-byte aligned");
  MIE_CHECK_ARG(!q || (scales && cols % 128 == 0 && scale_ld >= rows && ldq >= cols && ldq % 8 == 0),
                "fused quantisation needs cols %% 128 == 0 and scale storage");
  if (rows == 0) return MIE_OK;
  // Quantised, sixteen lanes a group and eight (us): 1024 x 1536 3.0 and 3.9, 4096 x 768 5.1 and 5.3, 300 x 9728 5.1 and 5.0,
  // 4096 x 1024 6.3 and 5.9, 4096 x 9728 57 and 45.
  const bool two = cols % 128 == 0 && (long long)rows * cols > 3 << 20;
  const RowBlocks shape(rows, cols / (two ? 16 : 8));
  MIE_CHECK_ARG(shape.blocks <= 0x7fffffff, "too many rows (%d)", rows);
  MIE_CUDA(launch_chained(two ? silu_mul_kernel<2> : silu_mul_kernel<1>, shape.grid(), shape.block(), 0,
                          (cudaStream_t)stream, (const __nv_bfloat16*)gate, (const __nv_bfloat16*)up, ld_in,
                          (__nv_bfloat16*)out, (uint8_t*)q, ldq, scales, scale_ld, rows, cols, shape.per_row));
  MIE_LAUNCH_CHECK("silu_mul_kernel");
  return MIE_OK;
}

extern "C" int mie_rope(mie_view4_t x, const void* cos, const void* sin, int64_t cs_batch_stride,
                        int64_t cs_token_stride, mie_view4_t out, int32_t batch, int32_t heads, int32_t seq,
                        int32_t dim, void* stream) {
  MIE_CHECK_ARG(x.ptr && cos && sin && out.ptr, "null pointer");
  MIE_CHECK_ARG(dim >= 2 && dim % 2 == 0 && x.stride[3] == 1 && out.stride[3] == 1, "RoPE needs an even, contiguous head_dim");
  const long long rows = (long long)batch * heads * seq;
  if (rows == 0) return MIE_OK;
  const int threads = 256;
  rope_kernel<<<(unsigned)((rows * 32 + threads - 1) / threads), threads, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x.ptr, x.stride[0], x.stride[1], x.stride[2], (const __nv_bfloat16*)cos,
      (const __nv_bfloat16*)sin, cs_batch_stride, cs_token_stride, (__nv_bfloat16*)out.ptr, out.stride[0],
      out.stride[1], out.stride[2], heads, seq, dim, rows);
  MIE_LAUNCH_CHECK("rope_kernel");
  return MIE_OK;
}

namespace {

int launch_qkv_post(mie::QkvParams& p, const void* qkv, int64_t ld, int32_t tokens, void* stream) {
  MIE_CHECK_ARG(qkv != nullptr && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(qkv) & 7) == 0,
                "qkv rows must be 8-byte aligned");
  if (tokens == 0) return MIE_OK;
  p.qkv = (const __nv_bfloat16*)qkv;
  p.ld = ld;
  auto rows16 = [](const void* ptr, const long long* strides) {
    return aligned16(ptr) && strides[0] % 8 == 0 && strides[1] % 8 == 0 && strides[2] % 8 == 0;
  };
  p.wide = ld % 8 == 0 && aligned16(qkv) && aligned16(p.q_weight) && aligned16(p.k_weight) && aligned16(p.cos_sin) &&
           aligned16(p.q_out) &&
           (p.kv8_pool != nullptr ? (reinterpret_cast<uintptr_t>(p.kv8_pool) & 7) == 0 && p.kv8_page_stride % 8 == 0
                                  : rows16(p.key_blocks, p.kb_s) && rows16(p.value_blocks, p.vb_s));
  const int lanes = ((p.q_heads + 2 * p.kv_heads) * 16 + 31) / 32 * 32;
  const int threads = lanes < 256 ? lanes : 256;
  // Few tokens: several blocks each, so that a half-warp has one head (one token of 48 heads 3 us less).
  const int blocks = tokens <= sm_count() ? (lanes + threads - 1) / threads : 1;
  MIE_CUDA(launch_chained(qkv_post_kernel, dim3((unsigned)tokens, (unsigned)blocks), dim3(threads), 0,
                          (cudaStream_t)stream, p));
  MIE_LAUNCH_CHECK("qkv_post_kernel");
  return MIE_OK;
}

}  // namespace

extern "C" int mie_qkv_norm_rope_write(const void* qkv, int64_t ld, const void* q_weight, const void* k_weight,
                                       const void* cos_sin, int32_t max_pos, mie_index_t positions,
                                       mie_index_t token_to_sequence, mie_index_t block_tables, void* q_out,
                                       mie_view4_t key_blocks, mie_view4_t value_blocks, int32_t tokens,
                                       int32_t q_heads, int32_t kv_heads, int32_t block_size, int32_t num_blocks,
                                       int32_t table_rows, int32_t table_width, float eps, int32_t* status,
                                       void* stream) {
  QkvParams p;
  if (int rc = qkv_bf16_pages(p, key_blocks, value_blocks)) return rc;
  if (int rc = qkv_common(p, q_weight, k_weight, cos_sin, max_pos, positions, token_to_sequence, block_tables, q_out,
                          tokens, q_heads, kv_heads, block_size, num_blocks, table_rows, table_width, eps, status))
    return rc;
  return launch_qkv_post(p, qkv, ld, tokens, stream);
}

extern "C" int mie_qkv_norm_rope_write_kv8(const void* qkv, int64_t ld, const void* q_weight, const void* k_weight,
                                           const void* cos_sin, int32_t max_pos, mie_index_t positions,
                                           mie_index_t token_to_sequence, mie_index_t block_tables, void* q_out,
                                           void* kv_pool, int64_t page_stride_bytes, float* kv_scales,
                                           int32_t tokens, int32_t q_heads, int32_t kv_heads, int32_t num_blocks,
                                           int32_t table_rows, int32_t table_width, float eps, int32_t* status,
                                           void* stream) {
  QkvParams p;
  if (int rc = qkv_e4m3_pool(p, kv_pool, page_stride_bytes, kv_scales, kv_heads)) return rc;
  if (int rc = qkv_common(p, q_weight, k_weight, cos_sin, max_pos, positions, token_to_sequence, block_tables, q_out,
                          tokens, q_heads, kv_heads, /*block_size=*/16, num_blocks, table_rows, table_width, eps, status))
    return rc;
  return launch_qkv_post(p, qkv, ld, tokens, stream);
}
