// What happens to a merged q/k/v row after its projection - q/k RMSNorm, RoPE, the K/V page write - shared by the kernel
// that reads projected rows (fused_glue.cu) and the projection that finishes its own (fp8_gemm.cu).
#pragma once

#include "common.cuh"
#include "glue.cuh"

namespace mie {

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool aligned8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }

struct QkvParams {
  const __nv_bfloat16* qkv;  // [tokens][ld]: q heads | k heads | v heads
  long long ld;
  const __nv_bfloat16* q_weight;
  const __nv_bfloat16* k_weight;
  const __nv_bfloat16* cos_sin;  // [max_pos][2][128]: cos row then sin row
  int max_pos;
  IndexView positions;           // [tokens]
  IndexView token_to_sequence;   // [tokens] or null (token t belongs to sequence t)
  IndexView tables;              // [sequences][width]
  __nv_bfloat16* q_out;          // [tokens][q_heads][128]
  char* key_blocks;
  char* value_blocks;
  long long kb_s[3], vb_s[3];    // page, head, token strides (elements)
  int tokens, q_heads, kv_heads, block_size, num_blocks, table_rows, table_width;
  float eps;
  int* status;
  // e4m3 K/V pool [pages][kv_heads][2][16][128] with scales [pages][kv_heads][2][16] (block_size 16), or null.
  uint8_t* kv8_pool;
  long long kv8_page_stride;  // bytes
  float* kv8_scales;
  bool wide;  // every row of every tensor is 16-byte aligned, of the e4m3 pool 8-byte (otherwise 8- and 4-byte)
};

// Where token t stands: its position and the page of its K / V rows, -1 when the metadata does not allow one (reported
// by the thread with `report`).
__device__ __forceinline__ void qkv_place(const QkvParams& p, int t, bool report, long long& pos, long long& page) {
  pos = p.positions.at(t);
  const long long seq = p.token_to_sequence.valid() ? p.token_to_sequence.at(t) : t;
  page = -1;
  if (report && (pos < 0 || pos >= p.max_pos)) raise_status(p.status, MIE_STATUS_BAD_POSITION);
  if (seq < 0 || seq >= p.table_rows) {
    if (report) raise_status(p.status, MIE_STATUS_BAD_SEQUENCE);
  } else if (pos < 0 || pos >= (long long)p.table_width * p.block_size) {
    if (report) raise_status(p.status, MIE_STATUS_BAD_POSITION);
  } else {
    page = p.tables.at(seq, pos / p.block_size);
    if (page < 0 || page >= p.num_blocks) {
      if (report) raise_status(p.status, MIE_STATUS_BAD_PAGE);
      page = -1;
    }
  }
}

// A head's sum of squares has one order of additions wherever a row is normed, so that a token's queries and keys do not
// depend on how many tokens share its step: four consecutive dims, then halves of the 32 fours 16, 8, 4, 2, 1 apart.
// Here 16 lanes hold eight dims each, two fours: the first exchange leaves every lane one four's sum, the last joins both
// (one exchange more than adding the eight first: 12032 tokens of 48 heads 1.3 % more).
__device__ __forceinline__ float half_warp_square_sum(const float (&v)[8], int l16) {
  const float low = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
  const float high = v[4] * v[4] + v[5] * v[5] + v[6] * v[6] + v[7] * v[7];
  const bool upper = (l16 & 8) != 0;
  float sum = (upper ? high : low) + __shfl_xor_sync(0xffffffffu, upper ? low : high, 8);
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  return sum + __shfl_xor_sync(0xffffffffu, sum, 8);
}

// One row of head slot h by a whole warp, four consecutive dims a lane (partner dims d +/- 64 sit 16 lanes away).
__device__ __forceinline__ void qkv_row_warp(const QkvParams& p, int t, int h, int lane, const uint2& raw, long long pos,
                                             long long page) {
  const bool is_q = h < p.q_heads, is_v = h >= p.q_heads + p.kv_heads;
  uint2 result = raw;
  if (!is_v) {
    const long long cpos = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
    const __nv_bfloat16* cs = p.cos_sin + cpos * 256 + lane * 4;
    float v[4], w[4], c[4], s[4], o[4];
    unpack4(*reinterpret_cast<const uint2*>(cs), c);
    unpack4(*reinterpret_cast<const uint2*>(cs + 128), s);
    unpack4(*reinterpret_cast<const uint2*>((is_q ? p.q_weight : p.k_weight) + lane * 4), w);
    unpack4(raw, v);
    const float ss = warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]);
    const float inv = rsqrtf(ss / 128.f + p.eps);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float n = round_bf16(w[j] * round_bf16(v[j] * inv));
      const float partner = __shfl_xor_sync(0xffffffffu, n, 16);
      const float rot = lane < 16 ? -partner : partner;  // rotate_half: (-x2, x1)
      o[j] = round_bf16(n * c[j]) + round_bf16(rot * s[j]);
    }
    result = pack4(o);
  }
  if (is_q) {
    *reinterpret_cast<uint2*>(p.q_out + ((long long)t * p.q_heads + h) * 128 + lane * 4) = result;
    return;
  }
  if (page < 0) return;
  const int kvh = is_v ? h - p.q_heads - p.kv_heads : h - p.q_heads, slot = (int)(pos % p.block_size);
  if (p.kv8_pool != nullptr) {
    float v[4];
    unpack4(result, v);
    const float amax = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    const float scale = __fdiv_rn(amax, 448.0f);
    uint32_t packed[1];
    quantize_values(v, fmaxf(scale, 1e-12f), packed);
    uint8_t* row = p.kv8_pool + page * p.kv8_page_stride + ((long long)kvh * 2 + (is_v ? 1 : 0)) * 2048 + slot * 128;
    *reinterpret_cast<uint32_t*>(row + lane * 4) = packed[0];
    if (lane == 0) p.kv8_scales[((page * p.kv_heads + kvh) * 2 + (is_v ? 1 : 0)) * 16 + slot] = scale;
    return;
  }
  const long long* st = is_v ? p.vb_s : p.kb_s;
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(is_v ? p.value_blocks : p.key_blocks) + page * st[0] +
                       (long long)kvh * st[1] + slot * st[2] + lane * 4;
  *reinterpret_cast<uint2*>(dst) = result;
}

// Host side: the cache (bf16 pages or the e4m3 pool), then everything else.
inline int qkv_bf16_pages(QkvParams& p, const mie_view4_t& key_blocks, const mie_view4_t& value_blocks) {
  MIE_CHECK_ARG(key_blocks.ptr && value_blocks.ptr, "null pointer");
  MIE_CHECK_ARG(aligned8(key_blocks.ptr) && aligned8(value_blocks.ptr), "pages must be 8-byte aligned");
  MIE_CHECK_ARG(key_blocks.stride[3] == 1 && value_blocks.stride[3] == 1, "pages must be contiguous in head_dim");
  for (int i = 0; i < 3; ++i) {
    MIE_CHECK_ARG(key_blocks.stride[i] % 4 == 0 && value_blocks.stride[i] % 4 == 0, "page strides must be multiples of 4");
    p.kb_s[i] = key_blocks.stride[i];
    p.vb_s[i] = value_blocks.stride[i];
  }
  p.key_blocks = (char*)key_blocks.ptr;
  p.value_blocks = (char*)value_blocks.ptr;
  p.kv8_pool = nullptr;
  p.kv8_page_stride = 0;
  p.kv8_scales = nullptr;
  return MIE_OK;
}

inline int qkv_e4m3_pool(QkvParams& p, void* kv_pool, int64_t page_stride_bytes, float* kv_scales, int32_t kv_heads) {
  MIE_CHECK_ARG(kv_pool && kv_scales, "null pointer");
  MIE_CHECK_ARG(page_stride_bytes >= (long long)kv_heads * 4096 && page_stride_bytes % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(kv_pool) | reinterpret_cast<uintptr_t>(kv_scales)) & 3) == 0,
                "the e4m3 pool needs a page stride of at least kv_heads * 4096 bytes, pool and scales 4-byte alignment");
  p.key_blocks = p.value_blocks = nullptr;
  for (int i = 0; i < 3; ++i) p.kb_s[i] = p.vb_s[i] = 0;
  p.kv8_pool = (uint8_t*)kv_pool;
  p.kv8_page_stride = page_stride_bytes;
  p.kv8_scales = kv_scales;
  return MIE_OK;
}

inline int qkv_common(QkvParams& p, const void* q_weight, const void* k_weight, const void* cos_sin, int32_t max_pos,
                      const mie_index_t& positions, const mie_index_t& token_to_sequence,
                      const mie_index_t& block_tables, void* q_out, int32_t tokens, int32_t q_heads, int32_t kv_heads,
                      int32_t block_size, int32_t num_blocks, int32_t table_rows, int32_t table_width, float eps,
                      int32_t* status) {
  MIE_CHECK_ARG(q_weight && k_weight && cos_sin && positions.ptr && block_tables.ptr && q_out, "null pointer");
  MIE_CHECK_ARG(aligned8(q_weight) && aligned8(k_weight) && aligned8(cos_sin) && aligned8(q_out),
                "norm weights, rotation table and query rows must be 8-byte aligned");
  MIE_CHECK_ARG(tokens >= 0 && q_heads >= 1 && kv_heads >= 1 && max_pos >= 1, "invalid shape");
  p.qkv = nullptr;
  p.ld = 0;
  p.q_weight = (const __nv_bfloat16*)q_weight;
  p.k_weight = (const __nv_bfloat16*)k_weight;
  p.cos_sin = (const __nv_bfloat16*)cos_sin;
  p.max_pos = max_pos;
  p.positions = IndexView(positions);
  p.token_to_sequence = IndexView(token_to_sequence);
  p.tables = IndexView(block_tables);
  p.q_out = (__nv_bfloat16*)q_out;
  p.tokens = tokens;
  p.q_heads = q_heads;
  p.kv_heads = kv_heads;
  p.block_size = block_size;
  p.num_blocks = num_blocks;
  p.table_rows = table_rows;
  p.table_width = table_width;
  p.eps = eps;
  p.status = status;
  p.wide = false;
  return MIE_OK;
}

}  // namespace mie
