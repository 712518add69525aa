// Projections of up to 128 rows in bf16: Y[m, n] = X[m, k] W[n, k]^T (+ bias[n]), fp32 accumulation.
//
// Such a product streams the weights once and does little else, and in a decode step it is one link of a chain of short
// kernels: besides HBM bandwidth the time between the end of the kernel before it and its own end counts.  Both kernels
// request their first weights before the launch-chain wait (the caller promises that no kernel queued before, however
// far back, writes them) and are launched in the same programmatic chain as the rest of the library.
//
//   * linear_rows_kernel, few rows: weights go from global memory straight into registers, as the A operand of mma.sync
//     (16 weight rows x 8 tokens).  A warp keeps D units of 16 rows x 64 columns in flight; a block of 8 warps takes 16
//     weight rows, warp w the units w, w + 8, ..., and the warps' sums meet in shared memory in warp order.  No ring, no
//     tensor memory, no cluster: after the wait only the activations (a few KB, in L2) are missing.
//   * linear_tile_kernel, more rows, where every block reading all activations would cost more L2 traffic than the
//     weights: 128 weight rows are the rows of a tcgen05 MMA, the tokens its BN columns, both staged by TMA, one fp32
//     accumulator in TMEM.  K is cut across a cluster of up to 8 CTAs, which read each other's parked sums and add them
//     in rank order.
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "umma.cuh"

namespace mie {
namespace {

struct LinearParams {
  const __nv_bfloat16* w;
  long long ldw;
  const __nv_bfloat16* x;
  long long ldx;
  int m, n, k;
  const __nv_bfloat16* bias;
  __nv_bfloat16* y;
  long long ldy;
  int* status;
  int prefetch;  // weights are requested before the launch-chain wait
};

// ---------------------------------------------------------------------------
// Few rows
// ---------------------------------------------------------------------------
constexpr int kRowsWarps = 8;
constexpr int kRowsTile = 16;  // weight rows of a block
constexpr int kRowsUnit = 64;  // columns of a unit

template <int NT>
constexpr int rows_depth() {
  return NT == 1 ? 4 : NT == 2 ? 3 : 2;
}

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// A lane (g = lane / 4, t = lane % 4) reads 16 bytes of rows g and g + 8, four lanes a row: 64 contiguous bytes of 8
// rows per load.  Its 8 values serve as the k slots 2t, 2t+1, 2t+8, 2t+9 of two MMAs; the activations are read in the
// same order, so that the permutation of k cancels.
template <int NT>
struct RowsUnit {
  uint4 a[4];       // rows g (columns 8t, 32 + 8t) and g + 8
  uint4 b[2 * NT];  // tokens 8 nt + g, the same columns
};

template <int NT>
__global__ void __launch_bounds__(kRowsWarps * 32, 2) linear_rows_kernel(const LinearParams p) {
  constexpr int D = rows_depth<NT>();
  constexpr int kTokens = 8 * NT;
  __shared__ float red[2][kRowsWarps][kRowsTile][kTokens + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int units = (p.k + kRowsUnit - 1) / kRowsUnit;
  const int tiles = (p.n + kRowsTile - 1) / kRowsTile;
  const int own = warp < units ? (units - warp + kRowsWarps - 1) / kRowsWarps : 0;  // units of a row this warp takes
  const int my_tiles = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total = own * my_tiles;
  RowsUnit<NT> ring[D];

  chain_release();
  if (!p.prefetch) chain_wait();

  auto load_weights = [&](RowsUnit<NT>& u, int tile, int unit) {
    const int col = unit * kRowsUnit + t * 8;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int row = tile * kRowsTile + g + 8 * half;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const bool in = row < p.n && col + c * 32 < p.k;
        u.a[2 * half + c] = in ? ld_stream(p.w + (long long)row * p.ldw + col + c * 32) : make_uint4(0, 0, 0, 0);
      }
    }
  };
  auto load_tokens = [&](RowsUnit<NT>& u, int unit) {
    const int col = unit * kRowsUnit + t * 8;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int tok = nt * 8 + g;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        u.b[2 * nt + c] = tok < p.m && col + c * 32 < p.k
                              ? *reinterpret_cast<const uint4*>(p.x + (long long)tok * p.ldx + col + c * 32)
                              : make_uint4(0, 0, 0, 0);
    }
  };
  int load_tile = blockIdx.x, load_unit = warp;  // the next unit to request
  auto advance = [&]() {
    load_unit += kRowsWarps;
    if (load_unit >= units) {
      load_unit = warp;
      load_tile += gridDim.x;
    }
  };
#pragma unroll
  for (int s = 0; s < D; ++s) {
    if (s < total) {
      load_weights(ring[s], load_tile, load_unit);
      advance();
    }
  }
  chain_wait();
  {
    int unit = warp;
#pragma unroll
    for (int s = 0; s < D; ++s) {
      if (s < total) load_tokens(ring[s], unit);
      unit = unit + kRowsWarps >= units ? warp : unit + kRowsWarps;
    }
  }

  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  int tile = blockIdx.x, parity = 0;
  // The warps' sums of a finished tile, added in warp order and stored.  Two buffers: a warp a tile ahead writes the
  // other one, and the barrier keeps it from being two ahead of a reader.
  auto finish_tile = [&]() {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        red[parity][warp][g + 8 * (i >> 1)][nt * 8 + 2 * t + (i & 1)] = acc[nt][i];
        acc[nt][i] = 0.f;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRowsTile * kTokens; i += kRowsWarps * 32) {
      const int row = i % kRowsTile, tok = i / kRowsTile;
      const int out = tile * kRowsTile + row;
      if (tok < p.m && out < p.n) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kRowsWarps; ++w) sum += red[parity][w][row][tok];
        if (p.bias != nullptr) sum += __bfloat162float(p.bias[out]);
        p.y[(long long)tok * p.ldy + out] = __float2bfloat16_rn(sum);
      }
    }
    parity ^= 1;
    tile += gridDim.x;
  };

  if (own == 0) {
    for (int i = 0; i < my_tiles; ++i) finish_tile();
    return;
  }
  int left = own;  // units of the current tile still to come
  for (int i0 = 0; i0 < total; i0 += D) {
#pragma unroll
    for (int s = 0; s < D; ++s) {
      if (i0 + s >= total) break;
      RowsUnit<NT>& u = ring[s];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 &top = u.a[c], &bottom = u.a[2 + c];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const uint4& b = u.b[2 * nt + c];
          Mma16816<__nv_bfloat16>::run(acc[nt], top.x, bottom.x, top.y, bottom.y, b.x, b.y);
          Mma16816<__nv_bfloat16>::run(acc[nt], top.z, bottom.z, top.w, bottom.w, b.z, b.w);
        }
      }
      if (i0 + s + D < total) {
        load_weights(u, load_tile, load_unit);
        load_tokens(u, load_unit);
        advance();
      }
      if (--left == 0) {
        finish_tile();
        left = own;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// More rows
// ---------------------------------------------------------------------------
constexpr int kTileThreads = 192;  // 4 epilogue warps, TMA producer, MMA issuer
constexpr int kTileRows = 128;     // weight rows of a tile
constexpr int kTileK = 64;         // columns of a stage: 128 bytes of bf16

template <int BN>
struct TileSmem {
  static constexpr int kStageBytes = kTileRows * 128 + BN * 128;
  static constexpr int kCtasPerSm = BN <= 64 ? 2 : 1;
  static constexpr int kStages = (kCtasPerSm == 2 ? 104 : 208) * 1024 / kStageBytes;
  static constexpr int kTotal = kStages * kStageBytes + (2 * kStages + 1) * 8 + 16 + 1024;
  static_assert(kStages * kStageBytes >= kTileRows * BN * 4, "the ring also parks the fp32 sums");
};

// Rank r of a cluster adds the tokens of its slice over the sums that every CTA has parked ([token][row]), in rank
// order.  A warp takes a token, a lane four weight rows; the loads of several tokens from all ranks are in flight
// together.
template <int kSplit>
__device__ __forceinline__ void reduce_slice(const LinearParams& p, uint32_t park, int rank, int tile, int warp,
                                             int lane) {
  constexpr int kBatch = 16 / kSplit;
  const int slice = (p.m + kSplit - 1) / kSplit;
  const int lo = rank * slice, hi = lo + slice < p.m ? lo + slice : p.m;
  const int out = tile * kTileRows + lane * 4;
  const bool vec = p.ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0 && out + 4 <= p.n;
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (p.bias != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (out + i < p.n) bias[i] = __bfloat162float(p.bias[out + i]);
  }
  for (int j0 = lo + warp; j0 < hi; j0 += 4 * kBatch) {
    float4 part[kBatch][kSplit];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int j = j0 + 4 * u < hi ? j0 + 4 * u : j0;
#pragma unroll
      for (int peer = 0; peer < kSplit; ++peer)
        part[u][peer] = ld_cluster_f4(park + (uint32_t)((j * kTileRows + lane * 4) * 4), (uint32_t)peer);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int j = j0 + 4 * u;
      float4 sum = part[u][0];
#pragma unroll
      for (int peer = 1; peer < kSplit; ++peer) {
        sum.x += part[u][peer].x;
        sum.y += part[u][peer].y;
        sum.z += part[u][peer].z;
        sum.w += part[u][peer].w;
      }
      if (j >= hi) break;
      __nv_bfloat16* dst = p.y + (long long)j * p.ldy + out;
      const float v[4] = {sum.x + bias[0], sum.y + bias[1], sum.z + bias[2], sum.w + bias[3]};
      if (vec) {
        *reinterpret_cast<uint2*>(dst) =
            make_uint2(Mma16816<__nv_bfloat16>::pack(v[0], v[1]), Mma16816<__nv_bfloat16>::pack(v[2], v[3]));
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (out + i < p.n) dst[i] = __float2bfloat16_rn(v[i]);
      }
    }
  }
}

// grid = (weight-row tiles, split), cluster = (1, split, 1): CTA `rank` takes the rank-th part of K.
template <int BN>
__global__ void __launch_bounds__(kTileThreads, TileSmem<BN>::kCtasPerSm)
    linear_tile_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                       const LinearParams p) {
  using S = TileSmem<BN>;
  constexpr int kStages = S::kStages;
  constexpr uint32_t kTmemCols = BN < 32 ? 32 : BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ring + kStages * S::kStageBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* done_bar = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int split = gridDim.y, rank = blockIdx.y, tile = blockIdx.x;
  const int kb_total = (p.k + kTileK - 1) / kTileK;
  const int kb_first = (int)((long long)kb_total * rank / split);
  const int kb_count = (int)((long long)kb_total * (rank + 1) / split) - kb_first;

  // Set-up and the first weights overlap the kernels queued before this one.
  int prefetched = 0;
  if (warp == 4 && lane == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    mbar_fence_init();
    const uint64_t policy = l2_evict_first_policy();
    for (; p.prefetch && prefetched < kb_count && prefetched < kStages; ++prefetched) {
      mbar_expect_tx(&full_bar[prefetched], S::kStageBytes);
      tma_load_2d_hint(ring + (size_t)prefetched * S::kStageBytes, &map_w, &full_bar[prefetched],
                       (kb_first + prefetched) * kTileK, tile * kTileRows, policy);
    }
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  chain_release();
  chain_wait();

  bool ok = true;
  const int row = warp * 32 + lane;  // of the tile (epilogue warps)
  float acc[BN];
  if (warp == 4) {
    if (lane == 0) {
      const uint64_t policy = l2_evict_first_policy();  // weights are streamed once per call
      for (int i = 0; i < kb_count; ++i) {
        const int s = i % kStages;
        uint8_t* dst = ring + (size_t)s * S::kStageBytes;
        if (i >= prefetched) {
          if (!mbar_wait_bounded(&empty_bar[s], ((i / kStages) & 1u) ^ 1u)) {
            raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
            break;
          }
          mbar_expect_tx(&full_bar[s], S::kStageBytes);
          tma_load_2d_hint(dst, &map_w, &full_bar[s], (kb_first + i) * kTileK, tile * kTileRows, policy);
        }
        tma_load_2d(dst + kTileRows * 128, &map_x, &full_bar[s], (kb_first + i) * kTileK, 0);
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    {
      constexpr uint32_t idesc = instr_desc_bf16(kTileRows, BN, 0, 0);
      for (int i = 0; i < kb_count; ++i) {
        const int s = i % kStages;
        if (!warp_wait_bounded(&full_bar[s], (i / kStages) & 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          break;
        }
        tc_fence_after();
        if (!elect_one()) continue;
        const uint32_t a = smem_u32(ring + (size_t)s * S::kStageBytes);
        const uint64_t da = smem_desc_k128(a), db = smem_desc_k128(a + kTileRows * 128);
#pragma unroll
        for (int k = 0; k < 4; ++k)  // 16 columns = 32 bytes each
          umma_f16(tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, i > 0 || k > 0 ? 1u : 0u);
        umma_commit(&empty_bar[s]);
      }
      __syncwarp();
      if (elect_one()) umma_commit(done_bar);  // the accumulator is complete, the ring idle
    }
    __syncwarp();
  } else {
    ok = mbar_wait_bounded(done_bar, 0);
    if (!ok) raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
    tc_fence_after();
    const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
    if constexpr (BN >= 32) {
#pragma unroll
      for (int c = 0; c < BN; c += 32) tmem_ld32(lane_addr + c, *reinterpret_cast<float(*)[32]>(&acc[c]));
    } else {
      tmem_ld16(lane_addr, *reinterpret_cast<float(*)[16]>(&acc[0]));
    }
    tmem_ld_wait();
    if (kb_count == 0) {
#pragma unroll
      for (int j = 0; j < BN; ++j) acc[j] = 0.f;
    }
  }

  if (split == 1) {
    const int out = tile * kTileRows + row;
    if (warp < 4 && out < p.n && ok) {
      const float bias = p.bias != nullptr ? __bfloat162float(p.bias[out]) : 0.f;
#pragma unroll
      for (int j = 0; j < BN; ++j)
        if (j < p.m) p.y[(long long)j * p.ldy + out] = __float2bfloat16_rn(acc[j] + bias);
    }
  } else {
    // Every CTA parks its sums [token][row] in its own, now idle, ring (a CTA whose wait ran out parks nothing useful;
    // the status word says so).
    const uint32_t park = smem_u32(ring);
    if (warp < 4) {
#pragma unroll
      for (int j = 0; j < BN; ++j)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(park + (uint32_t)((j * kTileRows + row) * 4)), "f"(acc[j])
                     : "memory");
    }
    cluster_sync_all();
    if (warp < 4) {
      if (split == 2)
        reduce_slice<2>(p, park, rank, tile, warp, lane);
      else if (split == 4)
        reduce_slice<4>(p, park, rank, tile, warp, lane);
      else
        reduce_slice<8>(p, park, rank, tile, warp, lane);
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while a peer may still read its sums
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct LinearMapKey {
  const void* ptr;
  long long rows, k, ld;
  int box_rows;
  bool operator==(const LinearMapKey& o) const {
    return ptr == o.ptr && rows == o.rows && k == o.k && ld == o.ld && box_rows == o.box_rows;
  }
};
struct LinearMapHash {
  size_t operator()(const LinearMapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr);
    for (long long v : {k.rows, k.k, k.ld, (long long)k.box_rows}) h = h * 1000003u ^ (size_t)v;
    return h;
  }
};

// 2-D bf16 tensor map [rows, k] (row stride ld elements), box 64 x box_rows, 128-byte swizzle.
int linear_map(const void* ptr, long long rows, long long k, long long ld, int box_rows, CUtensorMap* out) {
  static std::mutex mu;
  static std::unordered_map<LinearMapKey, CUtensorMap, LinearMapHash> cache;
  const LinearMapKey key{ptr, rows, k, ld, box_rows};
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return MIE_OK;
    }
  }
  const uint64_t dims[2] = {(uint64_t)k, (uint64_t)rows};
  const uint64_t strides[1] = {(uint64_t)ld * 2};
  const uint32_t box[2] = {(uint32_t)kTileK, (uint32_t)box_rows};
  const int rc = make_tensor_map(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
                                 CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != MIE_OK) return rc;
  std::lock_guard<std::mutex> lock(mu);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return MIE_OK;
}

template <int NT>
int launch_rows(const LinearParams& p, cudaStream_t stream) {
  const int tiles = (p.n + kRowsTile - 1) / kRowsTile, slots = 2 * sm_count();
  MIE_CUDA(launch_chained(linear_rows_kernel<NT>, dim3((unsigned)(tiles < slots ? tiles : slots)),
                          dim3(kRowsWarps * 32), 0, stream, p));
  MIE_LAUNCH_CHECK("linear_rows_kernel");
  return MIE_OK;
}

template <int BN>
int launch_tiles(const LinearParams& p, cudaStream_t stream) {
  using S = TileSmem<BN>;
  static bool configured[64] = {false};
  int dev = 0;
  MIE_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    MIE_CUDA(cudaFuncSetAttribute(linear_tile_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal));
    configured[dev] = true;
  }
  CUtensorMap mw, mx;
  if (int rc = linear_map(p.w, p.n, p.k, p.ldw, kTileRows, &mw)) return rc;
  if (int rc = linear_map(p.x, p.m, p.k, p.ldx, BN, &mx)) return rc;
  // K is cut (in powers of two) while the clusters surely fit one wave: a cluster needs its CTAs on SMs of one GPC, so
  // the last tenth of the slots cannot be counted on (96 tiles cut in 3 measured 16 us, in 2 11 us).
  const int tiles = (p.n + kTileRows - 1) / kTileRows, kb = (p.k + kTileK - 1) / kTileK;
  const int slots = S::kCtasPerSm * sm_count() * 9 / 10;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= slots && kb >= 4 * split) split *= 2;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)tiles, (unsigned)split, 1);
  config.blockDim = dim3(kTileThreads, 1, 1);
  config.dynamicSmemBytes = S::kTotal;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = (unsigned)split;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = chained_launch_enabled() ? 2 : 1;
  prefer_shared_carveout(reinterpret_cast<const void*>(linear_tile_kernel<BN>));
  MIE_CUDA(cudaLaunchKernelEx(&config, linear_tile_kernel<BN>, mw, mx, p));
  MIE_LAUNCH_CHECK("linear_tile_kernel");
  return MIE_OK;
}

}  // namespace
}  // namespace mie

using namespace mie;

extern "C" int mie_linear(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* bias, void* y,
                          int64_t ldy, int32_t m, int32_t n, int32_t k, int32_t kernel, int32_t* status, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  MIE_CHECK_ARG(x && w && y, "null pointer");
  MIE_CHECK_ARG(m >= 0 && m <= MIE_LINEAR_MAX_ROWS && n >= 1 && k >= 1, "invalid product %d x %d x %d", m, n, k);
  MIE_CHECK_ARG(k % 8 == 0 && ldx >= k && ldw >= k && ldy >= n, "k must be a multiple of 8 within the row strides");
  MIE_CHECK_ARG(ldx % 8 == 0 && ldw % 8 == 0 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0,
                "operand rows must be 16-byte aligned");
  const int prefetch = weight_prefetch_enabled() && !(kernel & MIE_LINEAR_NO_WEIGHT_PREFETCH);
  kernel &= ~MIE_LINEAR_NO_WEIGHT_PREFETCH;
  MIE_CHECK_ARG(kernel >= 0 && kernel <= 2 && (kernel != 1 || m <= 32), "unknown kernel %d for %d rows", kernel, m);
  if (m == 0) return MIE_OK;
  const LinearParams p{(const __nv_bfloat16*)w, ldw, (const __nv_bfloat16*)x, ldx, m, n, k, (const __nv_bfloat16*)bias,
                       (__nv_bfloat16*)y, ldy, status, prefetch};
  // The register kernel has the shorter start and end, the tensor-memory kernel the better stream and K cut in parts: at
  // one row (norm included, us) 256 x 2048 3.6 against 5.0, 4096 x 2048 6.4 / 6.5, 8192 x 2048 12.7 / 8.6, and of long
  // sums, which a block of the first goes through alone, 256 x 4096 7.4 / 6.2, 512 x 12288 22.6 / 11.4; at 16 rows
  // 2048 x 512 4.2 / 6.0, 2048 x 2048 7.9 / 7.0, 128 x 8192 18.4 / 9.0.
  const long long work = (long long)n * k;
  const bool few = k <= 2048 && ((m <= 8 && work <= 4096ll * 2048) || (m <= 16 && work <= 1024ll * 1024));
  if (kernel == 1 || (kernel == 0 && few)) {
    if (m <= 8) return launch_rows<1>(p, stream);
    if (m <= 16) return launch_rows<2>(p, stream);
    return launch_rows<4>(p, stream);
  }
  if (m <= 16) return launch_tiles<16>(p, stream);
  if (m <= 32) return launch_tiles<32>(p, stream);
  if (m <= 64) return launch_tiles<64>(p, stream);
  return launch_tiles<128>(p, stream);
}
