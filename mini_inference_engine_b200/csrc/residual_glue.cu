// Row kernels around the sublayers of a decoder that norms a sublayer's input and its output: the fused
// "norm the result, add it to the residual stream, norm the stream for the next sublayer", a tanh-gelu with an
// optional per-token table factor, a gated norm, and a soft cap of logits.  Residual stream, norms, gates and
// logits are fp32, the other rows bf16 or fp32 (`dtype`).
#include "glue.cuh"
#include "rows.cuh"

namespace mie {
namespace {

// ---------------------------------------------------------------------------
// x += alpha * rms_norm(y) * y_weight; then out = rms_norm(x) * next_weight, or out = x without a next weight.
// One CTA per row; x is updated in place.
// ---------------------------------------------------------------------------
struct ResidualParams {
  float* x;
  long long ldx;
  const void* y;
  long long ldy;
  const void* y_weight;
  float alpha;
  const void* next_weight;  // may be null
  void* out;                // may be null
  long long ldo;
  int cols;
  float eps;
};

// A thread's first kKept groups of VEC entries, one block width apart, stay in registers with their operands, which
// are all fetched before the first reduction; wider rows are read again.
constexpr int kKept = 2;

template <typename T, int VEC>
__global__ void __launch_bounds__(512) residual_norm_kernel(ResidualParams p) {
  __shared__ float red[2][32];
  chain_release();
  chain_wait();
  const int tid = threadIdx.x, step = blockDim.x * VEC;
  float* x = p.x + (long long)blockIdx.x * p.ldx;
  const T* y = reinterpret_cast<const T*>(p.y) + (long long)blockIdx.x * p.ldy;
  const T* yw = reinterpret_cast<const T*>(p.y_weight);
  const T* nw = p.out == nullptr ? nullptr : reinterpret_cast<const T*>(p.next_weight);
  float sums[kKept][VEC], ys[kKept][VEC], yws[kKept][VEC];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kKept; ++k) {
    const int c = (k * blockDim.x + tid) * VEC;
    if (c < p.cols) {
      Vec<T, VEC>::load(y + c, ys[k]);
      Vec<float, VEC>::load(x + c, sums[k]);
      Vec<T, VEC>::load(yw + c, yws[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < kKept; ++k)
    if ((k * (int)blockDim.x + tid) * VEC < p.cols)
#pragma unroll
      for (int j = 0; j < VEC; ++j) ss += ys[k][j] * ys[k][j];
  for (int c = (kKept * blockDim.x + tid) * VEC; c < p.cols; c += step) {
    float v[VEC];
    Vec<T, VEC>::load(y + c, v);
#pragma unroll
    for (int j = 0; j < VEC; ++j) ss += v[j] * v[j];
  }
  const float inv_y = p.alpha / sqrtf(block_sum(ss, red[0]) / (float)p.cols + p.eps);
  ss = 0.f;
#pragma unroll
  for (int k = 0; k < kKept; ++k) {
    const int c = (k * blockDim.x + tid) * VEC;
    if (c < p.cols) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        sums[k][j] += ys[k][j] * inv_y * yws[k][j];
        ss += sums[k][j] * sums[k][j];
      }
      Vec<float, VEC>::store(x + c, sums[k]);
    }
  }
  for (int c = (kKept * blockDim.x + tid) * VEC; c < p.cols; c += step) {
    float v[VEC], w[VEC], r[VEC];
    Vec<T, VEC>::load(y + c, v);
    Vec<T, VEC>::load(yw + c, w);
    Vec<float, VEC>::load(x + c, r);
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      r[j] += v[j] * inv_y * w[j];
      ss += r[j] * r[j];
    }
    Vec<float, VEC>::store(x + c, r);
  }
  if (p.out == nullptr) return;
  const float inv_x = nw == nullptr ? 1.f : 1.f / sqrtf(block_sum(ss, red[1]) / (float)p.cols + p.eps);
  T* out = reinterpret_cast<T*>(p.out) + (long long)blockIdx.x * p.ldo;
  auto emit = [&](int c, float (&v)[VEC]) {
    if (nw != nullptr) {
      float w[VEC];
      Vec<T, VEC>::load(nw + c, w);
#pragma unroll
      for (int j = 0; j < VEC; ++j) v[j] = v[j] * inv_x * w[j];
    }
    Vec<T, VEC>::store(out + c, v);
  };
#pragma unroll
  for (int k = 0; k < kKept; ++k) {
    const int c = (k * blockDim.x + tid) * VEC;
    if (c < p.cols) emit(c, sums[k]);
  }
  for (int c = (kKept * blockDim.x + tid) * VEC; c < p.cols; c += step) {
    float v[VEC];
    Vec<float, VEC>::load(x + c, v);
    emit(c, v);
  }
}

// ---------------------------------------------------------------------------
// out = gelu(in) (* table[ids[row]][c]), gelu(z) = z / 2 (1 + tanh(sqrt(2 / pi) (z + 0.044715 z^3))).
// ---------------------------------------------------------------------------
struct GeluParams {
  const void* in;
  long long ld_in;
  IndexView ids;  // with the table
  const void* table;
  long long ld_table, vocab;
  void* out;
  long long ldo;
  int rows, cols;
  int* status;
};

__device__ __forceinline__ float gelu_tanh(float z) {
  const float inner = 0.7978845608028654f * (z + 0.044715f * z * z * z);
  return 0.5f * z * (1.f + tanhf(inner));
}

// The same as z / (1 + exp(-2 inner)) with the approximate exponential and reciprocal, for 16-bit results, and without the
// cancellation of 1 + tanh at negative z.  The error is that of the exponent, four or five roundings of a number that grows
// with z: 2^-21 at |z| <= 1, 2^-17 at -9.  Against 64 bits, over all bf16 z in [-10, 10] and 200 factors of a table each, 31 of
// 1.2 million results are rounded to the other side (all by a tie's width, 0.5003 units), with tanhf 29,092, up to 256 units
// off.  Below -10 the result is -0, where it would be 1e-37 and less.
__device__ __forceinline__ float gelu_tanh16(float z) {
  const float inner = 0.7978845608028654f * (z + 0.044715f * z * z * z);
  return gate_quotient(z, gate_denominator(inner * (-2.f * kLog2e)));
}

// Bound by HBM (4 bytes an entry in bf16) with few instructions: tanhf and a 64-bit index division an item took 10000 x 6144
// 67 us, now 53 (64 x 12288 2.6 and 2.1).
template <typename T, int VEC>
__global__ void gelu_kernel(GeluParams p, int blocks_per_row) {
  chain_release();
  chain_wait();
  const int first = blockIdx.x / blocks_per_row;
  const long long row = (long long)first * blockDim.y + threadIdx.y;
  const int c = (int)((blockIdx.x - first * blocks_per_row) * blockDim.x + threadIdx.x) * VEC;
  if (row >= p.rows || c >= p.cols) return;
  float v[VEC];
  Vec<T, VEC>::load(reinterpret_cast<const T*>(p.in) + row * p.ld_in + c, v);
#pragma unroll
  for (int j = 0; j < VEC; ++j) v[j] = sizeof(T) == 2 ? gelu_tanh16(v[j]) : gelu_tanh(v[j]);
  if (p.table != nullptr) {
    long long id = p.ids.at(row);
    if (id < 0 || id >= p.vocab) {
      if (c == 0) raise_status(p.status, MIE_STATUS_BAD_TOKEN);
      id = 0;
    }
    float e[VEC];
    Vec<T, VEC>::load(reinterpret_cast<const T*>(p.table) + id * p.ld_table + c, e);
#pragma unroll
    for (int j = 0; j < VEC; ++j) v[j] *= e[j];
  }
  Vec<T, VEC>::store(reinterpret_cast<T*>(p.out) + row * p.ldo + c, v);
}

// ---------------------------------------------------------------------------
// out = rms_norm(x) * weight * sigmoid(gate).  One CTA per row.
// ---------------------------------------------------------------------------
struct GatedNormParams {
  const void* x;
  long long ldx;
  const void* gate;
  long long ldg;
  const void* weight;
  void* out;
  long long ldo;
  int cols;
  float eps;
};

template <typename T, int VEC>
__global__ void __launch_bounds__(512) gated_norm_kernel(GatedNormParams p) {
  __shared__ float red[32];
  chain_release();
  chain_wait();
  const int tid = threadIdx.x, step = blockDim.x * VEC;
  const T* x = reinterpret_cast<const T*>(p.x) + (long long)blockIdx.x * p.ldx;
  const T* gate = reinterpret_cast<const T*>(p.gate) + (long long)blockIdx.x * p.ldg;
  T* out = reinterpret_cast<T*>(p.out) + (long long)blockIdx.x * p.ldo;
  const T* weight = reinterpret_cast<const T*>(p.weight);
  float xs[kKept][VEC], ws[kKept][VEC], gs[kKept][VEC];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kKept; ++k) {
    const int c = (k * blockDim.x + tid) * VEC;
    if (c < p.cols) {
      Vec<T, VEC>::load(x + c, xs[k]);
      Vec<T, VEC>::load(weight + c, ws[k]);
      Vec<T, VEC>::load(gate + c, gs[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < kKept; ++k)
    if ((k * (int)blockDim.x + tid) * VEC < p.cols)
#pragma unroll
      for (int j = 0; j < VEC; ++j) ss += xs[k][j] * xs[k][j];
  for (int c = (kKept * blockDim.x + tid) * VEC; c < p.cols; c += step) {
    float v[VEC];
    Vec<T, VEC>::load(x + c, v);
#pragma unroll
    for (int j = 0; j < VEC; ++j) ss += v[j] * v[j];
  }
  const float inv = 1.f / sqrtf(block_sum(ss, red) / (float)p.cols + p.eps);
  auto emit = [&](int c, float (&v)[VEC], const float (&w)[VEC], const float (&g)[VEC]) {
#pragma unroll
    for (int j = 0; j < VEC; ++j) v[j] = __fdividef(v[j] * inv * w[j], 1.f + expf(-g[j]));
    Vec<T, VEC>::store(out + c, v);
  };
#pragma unroll
  for (int k = 0; k < kKept; ++k) {
    const int c = (k * blockDim.x + tid) * VEC;
    if (c < p.cols) emit(c, xs[k], ws[k], gs[k]);
  }
  for (int c = (kKept * blockDim.x + tid) * VEC; c < p.cols; c += step) {
    float v[VEC], w[VEC], g[VEC];
    Vec<T, VEC>::load(x + c, v);
    Vec<T, VEC>::load(weight + c, w);
    Vec<T, VEC>::load(gate + c, g);
    emit(c, v, w, g);
  }
}

// logits <- cap * tanh(logits / cap), in place, 16 bytes a thread from the first aligned element on (one element a thread:
// 64 x 151936 41 us, now 13.7).
__global__ void softcap_kernel(float* logits, long long count, float cap, int head) {
  chain_release();
  chain_wait();
  auto capped = [&](float x) { return cap * tanhf(x / cap); };
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = head + t * 4;
  if (t < head) logits[t] = capped(logits[t]);
  if (i + 4 <= count) {
    float4 v = *reinterpret_cast<const float4*>(logits + i);
    *reinterpret_cast<float4*>(logits + i) = make_float4(capped(v.x), capped(v.y), capped(v.z), capped(v.w));
  } else {
    for (long long j = i; j < count; ++j) logits[j] = capped(logits[j]);
  }
}

// Greedy token of a row: index of its largest value, the first one among equals; a NaN counts as larger than any number.
// A cluster of CTAs reads a row in 16-byte pieces, each thread keeping its best, and the first CTA compares the others'.
constexpr int kArgmaxCtas = 8, kArgmaxThreads = 256;

__device__ __forceinline__ unsigned long long argmax_key(float v, int index) {
  const uint32_t bits = __float_as_uint(v);
  const uint32_t order = v != v ? 0xffffffffu : bits >> 31 ? ~bits : bits | 0x80000000u;
  return (unsigned long long)(v == 0.f ? 0x80000000u : order) << 32 | (uint32_t)~index;
}

template <typename T>
__global__ void __cluster_dims__(kArgmaxCtas, 1, 1) __launch_bounds__(kArgmaxThreads)
    argmax_rows_kernel(const T* logits, long long ld, int cols, int vec, long long* out) {
  __shared__ unsigned long long best_of[kArgmaxThreads / 32];
  chain_release();
  chain_wait();
  constexpr int kVec = 16 / (int)sizeof(T), kBatch = 4;
  const int row = blockIdx.x / kArgmaxCtas, rank = blockIdx.x % kArgmaxCtas, step = kArgmaxCtas * kArgmaxThreads;
  const T* src = logits + (long long)row * ld;
  const int first = rank * kArgmaxThreads + threadIdx.x, units = vec ? cols / kVec : 0;
  unsigned long long best = 0;
  auto take = [&](float v, int index) {
    const unsigned long long key = argmax_key(v, index);
    best = key > best ? key : best;
  };
  for (int u0 = first; u0 < units; u0 += kBatch * step) {
    uint4 raw[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
      raw[b] = *reinterpret_cast<const uint4*>(src + (long long)(u0 + b * step < units ? u0 + b * step : u0) * kVec);
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int u = u0 + b * step < units ? u0 + b * step : u0;
      const T* v = reinterpret_cast<const T*>(&raw[b]);
#pragma unroll
      for (int i = 0; i < kVec; ++i) take(to_float<T>(v[i]), u * kVec + i);
    }
  }
  for (int c = units * kVec + first; c < cols; c += step) take(to_float<T>(src[c]), c);
  auto reduce = [](unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
      v = other > v ? other : v;
    }
    return v;
  };
  best = reduce(best);
  if ((threadIdx.x & 31) == 0) best_of[threadIdx.x >> 5] = best;
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank == 0 && threadIdx.x < 32) {
    constexpr int kWarps = kArgmaxThreads / 32;
    best = 0;
    for (int i = threadIdx.x; i < kArgmaxCtas * kWarps; i += 32) {
      uint32_t remote;
      unsigned long long v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&best_of[i % kWarps])), "r"(i / kWarps));
      asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
      best = v > best ? v : best;
    }
    best = reduce(best);
    if (threadIdx.x == 0) out[row] = (long long)(uint32_t)~(uint32_t)best;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

int row_threads(int cols, bool vec) {
  const int groups = vec ? cols / 8 : cols;
  const int threads = ((groups + kKept - 1) / kKept + 31) / 32 * 32;
  return threads > 512 ? 512 : threads;
}

// One CTA per row, in the vector width the rows allow.
#define MIE_LAUNCH_ROWS(kernel, dtype, rows, cols, vec, params)                                                     \
  do {                                                                                                              \
    const dim3 grid__((unsigned)(rows)), block__((unsigned)row_threads(cols, vec));                                 \
    if ((dtype) == MIE_DTYPE_BF16)                                                                                  \
      MIE_CUDA(vec ? launch_chained(kernel<__nv_bfloat16, 8>, grid__, block__, 0, (cudaStream_t)stream, params)     \
                   : launch_chained(kernel<__nv_bfloat16, 1>, grid__, block__, 0, (cudaStream_t)stream, params));   \
    else                                                                                                            \
      MIE_CUDA(vec ? launch_chained(kernel<float, 8>, grid__, block__, 0, (cudaStream_t)stream, params)             \
                   : launch_chained(kernel<float, 1>, grid__, block__, 0, (cudaStream_t)stream, params));           \
    MIE_LAUNCH_CHECK(#kernel);                                                                                      \
  } while (0)

}  // namespace
}  // namespace mie

using namespace mie;

extern "C" int mie_residual_norm(float* x, int64_t ldx, const void* y, int64_t ldy, const void* y_weight, float alpha,
                                 const void* next_weight, void* out, int64_t ldo, int32_t rows, int32_t cols,
                                 int32_t dtype, float eps, void* stream) {
  MIE_CHECK_ACT_DTYPE(dtype);
  MIE_CHECK_ARG(x && y && y_weight, "null pointer");
  MIE_CHECK_ARG(!next_weight || out, "a next norm needs an output");
  MIE_CHECK_ARG(rows >= 0 && cols >= 1, "invalid sizes");
  if (rows == 0) return MIE_OK;
  const ResidualParams p{x, ldx, y, ldy, y_weight, alpha, next_weight, out, ldo, cols, eps};
  const bool vec = cols % 8 == 0 && ldx % 4 == 0 && ldy % 8 == 0 && ldo % 8 == 0 && aligned(x, 16) && aligned(y, 16) &&
                   aligned(y_weight, 16) && aligned(next_weight, 16) && aligned(out, 16);
  MIE_LAUNCH_ROWS(residual_norm_kernel, dtype, rows, cols, vec, p);
  return MIE_OK;
}

extern "C" int mie_gelu(const void* in, int64_t ld_in, mie_index_t ids, const void* table, int64_t ld_table,
                        int64_t vocab, void* out, int64_t ldo, int32_t rows, int32_t cols, int32_t dtype,
                        int32_t* status, void* stream) {
  MIE_CHECK_ACT_DTYPE(dtype);
  MIE_CHECK_ARG(in && out, "null pointer");
  MIE_CHECK_ARG(!table || (ids.ptr && vocab >= 1), "a table factor needs token ids and the table's size");
  MIE_CHECK_ARG(rows >= 0 && cols >= 1, "invalid sizes");
  if (rows == 0) return MIE_OK;
  const GeluParams p{in, ld_in, IndexView(ids), table, ld_table, vocab, out, ldo, rows, cols, status};
  const bool vec = cols % 8 == 0 && ld_in % 8 == 0 && ldo % 8 == 0 && aligned(in, 16) && aligned(out, 16) &&
                   (!table || (ld_table % 8 == 0 && aligned(table, 16)));
  const RowBlocks shape(rows, vec ? cols / 8 : cols);
  MIE_CHECK_ARG(shape.blocks <= 0x7fffffff, "too many rows (%d)", rows);
  const dim3 grid = shape.grid(), block = shape.block();
  const int per_row = shape.per_row;
  if (dtype == MIE_DTYPE_BF16)
    MIE_CUDA(vec ? launch_chained(gelu_kernel<__nv_bfloat16, 8>, grid, block, 0, (cudaStream_t)stream, p, per_row)
                 : launch_chained(gelu_kernel<__nv_bfloat16, 1>, grid, block, 0, (cudaStream_t)stream, p, per_row));
  else
    MIE_CUDA(vec ? launch_chained(gelu_kernel<float, 8>, grid, block, 0, (cudaStream_t)stream, p, per_row)
                 : launch_chained(gelu_kernel<float, 1>, grid, block, 0, (cudaStream_t)stream, p, per_row));
  MIE_LAUNCH_CHECK("gelu_kernel");
  return MIE_OK;
}

extern "C" int mie_gated_norm(const void* x, int64_t ldx, const void* gate, int64_t ldg, const void* weight, void* out,
                              int64_t ldo, int32_t rows, int32_t cols, int32_t dtype, float eps, void* stream) {
  MIE_CHECK_ACT_DTYPE(dtype);
  MIE_CHECK_ARG(x && gate && weight && out, "null pointer");
  MIE_CHECK_ARG(rows >= 0 && cols >= 1, "invalid sizes");
  if (rows == 0) return MIE_OK;
  const GatedNormParams p{x, ldx, gate, ldg, weight, out, ldo, cols, eps};
  const bool vec = cols % 8 == 0 && ldx % 8 == 0 && ldg % 8 == 0 && ldo % 8 == 0 && aligned(x, 16) &&
                   aligned(gate, 16) && aligned(weight, 16) && aligned(out, 16);
  MIE_LAUNCH_ROWS(gated_norm_kernel, dtype, rows, cols, vec, p);
  return MIE_OK;
}

extern "C" int mie_softcap(float* logits, int64_t count, float cap, void* stream) {
  MIE_CHECK_ARG(logits && count >= 0 && cap > 0.f, "soft cap needs logits and a positive cap");
  if (count == 0) return MIE_OK;
  const int head = (int)(((16 - (reinterpret_cast<uintptr_t>(logits) & 15)) & 15) / 4);  // up to the first aligned one
  const long long threads = count / 4 + 4;  // also covers a row shorter than the head
  MIE_CUDA(launch_chained(softcap_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, (cudaStream_t)stream,
                          logits, (long long)count, cap, head < count ? head : (int)count));
  MIE_LAUNCH_CHECK("softcap_kernel");
  return MIE_OK;
}

extern "C" int mie_argmax_rows(const void* logits, int64_t ld, int32_t dtype, int32_t rows, int32_t cols, int64_t* out,
                               void* stream) {
  MIE_CHECK_ACT_DTYPE(dtype);
  MIE_CHECK_ARG(logits && out && rows >= 0 && cols >= 1 && ld >= cols, "invalid sizes");
  MIE_CHECK_ARG(rows <= 0x7fffffff / kArgmaxCtas, "too many rows");
  if (rows == 0) return MIE_OK;
  const int act = dtype == MIE_DTYPE_BF16 ? 8 : 4;
  const int vec = ld % act == 0 && aligned(logits, 16) ? 1 : 0;
  const dim3 grid((unsigned)(rows * kArgmaxCtas)), block(kArgmaxThreads);
  if (dtype == MIE_DTYPE_BF16)
    MIE_CUDA(launch_chained(argmax_rows_kernel<__nv_bfloat16>, grid, block, 0, (cudaStream_t)stream,
                            (const __nv_bfloat16*)logits, (long long)ld, cols, vec, (long long*)out));
  else
    MIE_CUDA(launch_chained(argmax_rows_kernel<float>, grid, block, 0, (cudaStream_t)stream, (const float*)logits,
                            (long long)ld, cols, vec, (long long*)out));
  MIE_LAUNCH_CHECK("argmax_rows_kernel");
  return MIE_OK;
}
