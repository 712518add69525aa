// FP8 (e4m3 x e4m3) GEMM with 128x128 weight-block scales and per-token
// per-128-column activation scales, fp32 accumulation, bf16/fp16 output:
//
//   Y[m, n] = sum_kb ( sum_{k in kb} X8[m, k] * W8[n, k] ) * a_scale[m, kb] * w_scale[n / 128, kb]
//
// sm_100a design
//   * tcgen05.mma kind::f8f6f4 (UMMA 128 x BN x 32), operands staged in shared
//     memory by TMA (2-D tiled loads, 128-byte swizzle, no multicast), fp32
//     accumulators in tensor memory.
//   * The scales change every 128 columns of K, so each K block is accumulated
//     in its own TMEM buffer (a ring) and the promotion warps add it into fp32
//     registers with that block's scale (tcgen05.ld + FFMA) while the tensor
//     core already works on the next block.
//   * Two kernels.  Up to 128 tokens (decode): fp8_gemm_kernel, "swapped" - the
//     128 UMMA rows are weight rows and the BN = 16..128 columns are tokens, so
//     a handful of tokens still fills the tensor core's M and the kernel is a
//     pure weight-streaming (HBM-bound) loop; 4 or 8 promotion warps, one TMA
//     producer warp, two MMA-issuer warps.  Its rows can be finished in place of
//     stored: SiLU(gate) * up with the next GEMM's quantisation, or the q/k norm,
//     RoPE and cache write of a merged qkv projection (Finish).
//     More than 128 tokens: fp8_gemm_wide_kernel (described at its definition).
//   * A shape with fewer output tiles than SMs cuts the K range of every tile
//     into parts that run as one thread-block cluster and are reduced through
//     distributed shared memory in a fixed order (deterministic; no global
//     partials, no atomics, no spinning).
//   * Every mbarrier wait is bounded; a wait that runs out sets
//     MIE_STATUS_WAIT_TIMEOUT, the roles fall through to the common exit and
//     TMEM is released.
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "glue.cuh"
#include "qkv_rows.cuh"
#include "umma.cuh"

namespace mie {
namespace {

constexpr int kTileR = 128;  // UMMA M
constexpr int kBlockK = 128; // bytes of K per pipeline stage = one scale block
constexpr int kUmmaK = 32;   // fp8 elements per tcgen05.mma

__device__ __forceinline__ void epi_bar_sync(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// --------------------------------------------------------------------------
// Kernel
// --------------------------------------------------------------------------
struct GemmParams {
  int m, n, k;            // tokens, weight rows, reduction length
  const float* a_scale;   // [k_blocks][a_scale_ld]  (token scales, K-block major)
  int a_scale_ld;
  const float* w_scale;   // [ceil(n/128)][w_scale_ld]
  int w_scale_ld;
  void* y;                // [m][ldy] bf16 or fp16
  long long ldy;
  int out_f16;
  int* status;
  int prefetch;           // weights of the first K blocks are requested before the launch-chain wait (static weights)
  // Wide kernel only: this launch covers output tiles [tile_begin, tile_end).  late_wait: the launch-chain
  // wait is taken at the end of the kernel instead of the start (second launch of a two-launch GEMM, whose
  // inputs are already known to be complete because the first launch waited for them).
  // early_release: the next launch may start before this one's wait (not when it is the second launch of a
  // two-launch GEMM, which takes the first one's wait for its own).
  int tile_begin, tile_end, late_wait, early_release;
  int band;  // wide kernel: token tiles per band (see wide_item)
  // Finish::kSilu: the quantised result (y is not written).
  uint8_t* q;
  long long ldq;
  float* q_scales;
  int q_scale_ld;
};

// What the narrow kernel does with a finished row of 128 outputs of one token.
enum class Finish {
  kStore,  // bf16 / fp16 to y
  kSilu,   // weights [gate | up]: SiLU(gate) * up as e4m3 with one scale per token and 128 columns
  kQkv     // weights [q | k | v], heads of 128: q/k norm, RoPE, queries to q_out, keys and values to the cache
};

// Scale staging: per chunk of kChunkKb K blocks the promotion warps pull every
// scale product they will need into shared memory in one batch, so no
// global-memory latency sits between two K blocks.
template <int BN>
struct ScaleStage {
  static constexpr int kChunkKb = 32;
  static constexpr int kFloats = kChunkKb * BN;  // one a_scale * w_scale product per (K block, token)
};

// Promotion warps of fp8_gemm_kernel: one per TMEM lane quadrant, from 33 tokens two and for 128 columns four, which share the
// columns.  Four cost 0.2 to 0.4 us of start and barriers, which more than four K blocks a CTA pay (us, two and four a
// quadrant: 96 tokens of 2560 x 9728 13.5 and 12.9, of 6144 x 2560 9.4 and 9.2, of 1536 x 2560, five blocks, 6.8 and 6.8, 65
// 6.6 and 6.35; of 4096 x 2048, four blocks, 7.0 and 7.4).
constexpr int narrow_warps(int bn, int blocks) { return bn >= 128 && blocks > 4 ? 16 : bn >= 64 ? 8 : 4; }
constexpr int narrow_threads(int warps) { return (warps + 3) * 32; }

template <int BN>
struct GemmSmem {
  static constexpr int kStageBytes = kTileR * kBlockK + BN * kBlockK;
  static constexpr int kScaleBytes = ScaleStage<BN>::kFloats * 4;
  // Narrow column tiles (few tokens) use few registers: two CTAs share an SM, which halves the cost of a
  // partial last wave and doubles the TMA requests in flight per SM.  (At 64 columns two CTAs of four stages each
  // measured 6144 x 2560 10.3 us against 9.3 and 19456 x 2560 20.7 against the wide kernel's 18.2.)
  static constexpr int kCtasPerSm = BN <= 32 ? 2 : 1;
  static constexpr int kBudget = (kCtasPerSm == 2 ? 108 : 200) * 1024 - kScaleBytes;
  static constexpr int kStages = (kBudget / kStageBytes) > 12 ? 12 : (kBudget / kStageBytes);
  // Accumulator ring in TMEM: up to 8 BN-column buffers, so the MMA issuers can run several K blocks ahead of the
  // promotion, but not more buffers than stages (see done_bar).
  static constexpr int kAccMax = (512 / kCtasPerSm) / BN < kStages ? (512 / kCtasPerSm) / BN : kStages;
  static constexpr int kAcc = kAccMax >= 8 ? 8 : kAccMax >= 4 ? 4 : 2;
  static constexpr int kBarBytes = (2 * kStages + 8) * 8;
  static constexpr int kPlaceBytes = BN * 16;  // Finish::kQkv: position and page of the tokens
  static constexpr int kTotal = kStages * kStageBytes + kBarBytes + kScaleBytes + kPlaceBytes + 64 + 1024;
  static_assert(kTotal <= (kCtasPerSm == 2 ? 113 : 226) * 1024, "shared memory of an SM");
  static_assert(kStages * kStageBytes >= BN * kTileR * 4, "the stage ring also parks the fp32 rows");
};

// Four outputs of a token from weight row n0 of the narrow kernel.
__device__ __forceinline__ void store_row4(const GemmParams& p, int tok, int n0, const float (&v)[4], bool vec) {
  uint16_t* dst = reinterpret_cast<uint16_t*>(p.y) + (long long)tok * p.ldy + n0;
  if (vec && n0 + 4 <= p.n) {
    uint2 w;
    w.x = p.out_f16 ? Mma16816<__half>::pack(v[0], v[1]) : Mma16816<__nv_bfloat16>::pack(v[0], v[1]);
    w.y = p.out_f16 ? Mma16816<__half>::pack(v[2], v[3]) : Mma16816<__nv_bfloat16>::pack(v[2], v[3]);
    *reinterpret_cast<uint2*>(dst) = w;
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (n0 + j >= p.n) break;
    if (p.out_f16)
      reinterpret_cast<__half*>(dst)[j] = __float2half_rn(v[j]);
    else
      reinterpret_cast<__nv_bfloat16*>(dst)[j] = __float2bfloat16_rn(v[j]);
  }
}

// The end of the narrow kernel.  Every CTA of the cluster has parked its fp32 sums as [token][128 weight rows]; CTA
// `rank` finishes its share of the live tokens.  A warp takes a token, a lane four weight rows (16-byte
// distributed-shared-memory loads, the rows of several tokens from all CTAs in flight together; none for tokens past the
// share: 33 tokens of 4096 x 2048 5.8 -> 5.4 us) and adds the kSplit
// parts of K in part order, so that results do not depend on timing.
template <int kWarps, int BN, Finish kFinish, int kSplit>
__device__ __forceinline__ void finish_rows(const GemmParams& p, const QkvParams& qkv, const longlong2* place,
                                            uint32_t park, int rank, int tile, int tok0, int warp, int lane) {
  constexpr int kPeers = kFinish == Finish::kSilu ? 2 * kSplit : kSplit;  // gate parts have even ranks, up parts odd ones
  constexpr int kBatch = kPeers >= 8 ? 1 : kPeers >= 4 ? 2 : 4;
  const int live = p.m - tok0 < BN ? p.m - tok0 : BN;
  const int slice = (live + kPeers - 1) / kPeers;
  const int lo = rank * slice, hi = lo + slice < live ? lo + slice : live;
  const bool vec = p.ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0;
  for (int j0 = lo + warp; j0 < hi; j0 += kWarps * kBatch) {
    float4 part[kBatch][kPeers];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int j = j0 + u * kWarps;
      if (j >= hi) break;
#pragma unroll
      for (int peer = 0; peer < kPeers; ++peer)
        part[u][peer] = ld_cluster_f4(park + (uint32_t)((j * kTileR + lane * 4) * 4), (uint32_t)peer);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int j = j0 + u * kWarps, tok = tok0 + j;
      if (j >= hi) break;
      auto total = [&](int first, int step, float (&v)[4]) {
        v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll
        for (int peer = first; peer < kPeers; peer += step) {
          v[0] += part[u][peer].x;
          v[1] += part[u][peer].y;
          v[2] += part[u][peer].z;
          v[3] += part[u][peer].w;
        }
      };
      float v[4];
      if constexpr (kFinish == Finish::kStore) {
        total(0, 1, v);
        store_row4(p, tok, tile * kTileR + lane * 4, v, vec);
      } else if constexpr (kFinish == Finish::kQkv) {
        total(0, 1, v);
        qkv_row_warp(qkv, tok, tile, lane, pack4(v), place[j].x, place[j].y);
      } else {
        // The rounding points of the unfused chain: gate and up to bf16, SiLU to bf16, their product to bf16.
        float up[4];
        total(0, 2, v);
        total(1, 2, up);
        uint2 raw;
        const uint2 up2 = pack4(up);
        __nv_bfloat162* r2 = reinterpret_cast<__nv_bfloat162*>(&raw);
        const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&up2);
#pragma unroll
        for (int i = 0; i < 2; ++i)
          r2[i] = __hmul2(__floats2bfloat162_rn(silu16(round_bf16(v[2 * i])), silu16(round_bf16(v[2 * i + 1]))),
                          u2[i]);
        unpack4(raw, v);
        const float amax = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
        const float scale = __fdiv_rn(amax, 448.0f);
        uint32_t packed[1];
        quantize_values(v, fmaxf(scale, 1e-12f), packed);
        *reinterpret_cast<uint32_t*>(p.q + (long long)tok * p.ldq + tile * kTileR + lane * 4) = packed[0];
        if (lane == 0) p.q_scales[(long long)tile * p.q_scale_ld + tok] = scale;
      }
    }
  }
}

// Up to 128 tokens.  The 128 UMMA rows are weight rows (one 128-row scale block per tile), the BN columns
// are tokens.  Warps 0..E-1 promote, warp E is the TMA producer, warps E + 1 and E + 2 issue the MMAs of alternate K blocks (one
// thread's wait, four MMAs and commit take about 770 cycles whatever BN is, and with a second commit per block 900:
// longer than the block's weights take from HBM) and the first of them owns TMEM.  A K block has one commit, on the barrier that
// both frees its stage and hands its accumulator to the promotion.
// grid = (tiles, split), cluster = (1, split, 1): CTA `rank` of a cluster takes the rank-th part of K.  Finish::kSilu: a
// cluster has a CTA for the gate rows and one for the up rows of every part of K (ranks 2 part and 2 part + 1).
template <int BN, Finish kFinish, int E>
__global__ void __launch_bounds__(narrow_threads(E), GemmSmem<BN>::kCtasPerSm)
    fp8_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ GemmParams p, const __grid_constant__ QkvParams qkv) {
  using S = GemmSmem<BN>;
  using SS = ScaleStage<BN>;
  constexpr int kCols = BN * 4 / E;  // columns of a promotion warp
  constexpr int kStages = S::kStages;
  constexpr int kAcc = S::kAcc;
  constexpr uint32_t kTmemCols = kAcc * BN < 32 ? 32 : kAcc * BN;
  static_assert((kTmemCols & (kTmemCols - 1)) == 0 && kTmemCols <= 512, "TMEM columns must be a power of two <= 512");
  static_assert(BN % 16 == 0, "token tile must be a multiple of 16");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* stage_base = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * S::kStageBytes);
  // The MMAs of the stage's K block have completed: waited for by the producer and, before the block after next of the
  // same stage can complete (kAcc <= kStages), by the promotion.
  uint64_t* done_bar = full_bar + kStages;
  uint64_t* tmem_empty = done_bar + kStages;
  float* sscale = reinterpret_cast<float*>(tmem_empty + 8);  // staged scale products of the current K chunk
  longlong2* place = reinterpret_cast<longlong2*>(sscale + SS::kFloats);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(place + BN);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int kb_total = (p.k + kBlockK - 1) / kBlockK;
  constexpr bool kPairs = kFinish == Finish::kSilu;
  const int tiles_n = (p.n + kTileR - 1) / kTileR / (kPairs ? 2 : 1);  // output tiles over the weight rows
  const int split = gridDim.y / (kPairs ? 2 : 1), rank = blockIdx.y, part = rank / (kPairs ? 2 : 1);
  const int tn = (int)blockIdx.x % tiles_n, tt = (int)blockIdx.x / tiles_n;  // output tile, token tile
  const int tw = kPairs && (rank & 1) ? tiles_n + tn : tn;                   // weight-row tile
  const int kb_first = (int)((long long)kb_total * part / split);
  const int kb_last = (int)((long long)kb_total * (part + 1) / split);  // exclusive

  // Everything up to the launch-chain wait overlaps the kernels queued before this one.  So does the weight half of
  // the first stages when the caller promises that none of those kernels writes the weights: the producer requests it
  // before the TMEM allocation, which may have to wait for an earlier kernel's, and adds the activation half after
  // the wait.
  uint32_t prefetched = 0;
  if (warp == E && lane == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&done_bar[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) mbar_init(&tmem_empty[b], E);
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
    if (p.prefetch) {
      const uint64_t stream_policy = l2_evict_first_policy();
      for (int kb = kb_first; kb < kb_last && prefetched < (uint32_t)kStages; ++kb, ++prefetched) {
        mbar_expect_tx(&full_bar[prefetched], S::kStageBytes);
        tma_load_2d_hint(stage_base + (size_t)prefetched * S::kStageBytes, &map_w, &full_bar[prefetched], kb * kBlockK,
                         tw * kTileR, stream_policy);
      }
    }
  }
  if (warp == E + 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_release();
  chain_wait();

  // Promotion state that outlives the role branch (the parked rows below need it).
  constexpr int kEpiThreads = E * 32;
  const int row_in_tile = (warp & 3) * 32 + lane, col0 = E == 4 ? 0 : (warp >> 2) * kCols;
  float acc[kCols];

  if (warp == E) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint64_t stream_policy = l2_evict_first_policy();  // weights are streamed once per call
      uint32_t n = 0;
      for (int kb = kb_first; kb < kb_last; ++kb, ++n) {
        const int s = n % kStages;
        uint8_t* dst = stage_base + (size_t)s * S::kStageBytes;
        if (n < prefetched) {  // the weight half is already on its way
          tma_load_2d(dst + kTileR * kBlockK, &map_x, &full_bar[s], kb * kBlockK, tt * BN);
          continue;
        }
        if (!mbar_wait_bounded(&done_bar[s], ((n / kStages) & 1u) ^ 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          break;
        }
        mbar_expect_tx(&full_bar[s], S::kStageBytes);
        tma_load_2d_hint(dst, &map_w, &full_bar[s], kb * kBlockK, tw * kTileR, stream_policy);
        tma_load_2d(dst + kTileR * kBlockK, &map_x, &full_bar[s], kb * kBlockK, tt * BN);
      }
    }
  } else if (warp > E) {
    // ---------------- MMA issuers ----------------
    {
      constexpr uint32_t idesc = instr_desc_f8(BN);
      const uint32_t blocks = (uint32_t)(kb_last - kb_first);
      for (uint32_t n = (uint32_t)(warp - (E + 1)); n < blocks; n += 2) {
        const int s = n % kStages, b = n % kAcc;
        // In this order: the stage's previous block may be the other issuer's, and a released accumulator (of a block no
        // older, kAcc <= kStages) tells that its barrier phase is over.
        if (!warp_wait_bounded(&tmem_empty[b], ((n / kAcc) & 1u) ^ 1u) ||
            !warp_wait_bounded(&full_bar[s], (n / kStages) & 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          break;
        }
        tc_fence_after();
        if (!elect_one()) continue;
        const uint32_t a_addr = smem_u32(stage_base + (size_t)s * S::kStageBytes);
        const uint32_t b_addr = a_addr + kTileR * kBlockK;
        const uint64_t da = smem_desc_k128(a_addr), db = smem_desc_k128(b_addr);
#pragma unroll
        for (int k = 0; k < kBlockK / kUmmaK; ++k) {
          umma_f8(tmem_base + b * BN, da + (uint64_t)(k * kUmmaK / 16), db + (uint64_t)(k * kUmmaK / 16), idesc,
                  k > 0 ? 1u : 0u);
        }
        umma_commit(&done_bar[s]);  // frees the smem stage and hands the accumulator to the promotion warps
      }
    }
  } else {
    // ---------------- Promotion warps: add every K block with its scales ----------------
    const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    const int epi_tid = threadIdx.x;  // promotion warps are warps 0..E-1
    if constexpr (kFinish == Finish::kQkv) {
      // The tokens' positions and pages, while the operands are on their way; the first output tile's CTA reports.
      if (epi_tid < BN && tt * BN + epi_tid < p.m) {
        long long pos, page;
        qkv_place(qkv, tt * BN + epi_tid, tn == 0 && rank == 0, pos, page);
        place[epi_tid] = make_longlong2(pos, page);
      }
    }
    uint32_t n = 0;
    bool ok = true;
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    for (int kb0 = kb_first; kb0 < kb_last && ok; kb0 += SS::kChunkKb) {
      const int kc = kb_last - kb0 < SS::kChunkKb ? kb_last - kb0 : SS::kChunkKb;
      // Stage this chunk's scale products a_scale[token] * w_scale (all loads in flight together).
      epi_bar_sync(kEpiThreads);  // the previous chunk's readers are done
      for (int i = epi_tid; i < kc * BN; i += kEpiThreads) {
        const int kk = i / BN, tok = tt * BN + i % BN;
        const float ws = p.w_scale[(long long)tw * p.w_scale_ld + kb0 + kk];
        sscale[i] = tok < p.m ? p.a_scale[(long long)(kb0 + kk) * p.a_scale_ld + tok] * ws : 0.f;
      }
      epi_bar_sync(kEpiThreads);
      for (int kk = 0; kk < kc; ++kk, ++n) {
        const int b = n % kAcc;
        const float* s_col = sscale + kk * BN + col0;
        if (!mbar_wait_bounded(&done_bar[n % kStages], (n / kStages) & 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t taddr = lane_addr + (uint32_t)(b * BN);
        if constexpr (kCols % 64 == 0) {
          // Two loads in flight per wait.
#pragma unroll
          for (int c = 0; c < kCols; c += 64) {
            float d0[32], d1[32];
            tmem_ld32(taddr + c, d0);
            tmem_ld32(taddr + c + 32, d1);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c + j] = fmaf(d0[j], s_col[c + j], acc[c + j]);
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c + 32 + j] = fmaf(d1[j], s_col[c + 32 + j], acc[c + 32 + j]);
          }
        } else if constexpr (kCols % 32 == 0) {
          float d[32];
          tmem_ld32(taddr, d);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = fmaf(d[j], s_col[j], acc[j]);
        } else {
          float d[16];
          tmem_ld16(taddr, d);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[j] = fmaf(d[j], s_col[j], acc[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[b]);
      }
    }
  }

  // ---------------- output ----------------
  // Every MMA of this CTA has completed (the promotion consumed the last accumulator), so the stage ring is free and
  // parks the rows.
  const uint32_t park = smem_u32(stage_base);
  if (warp < E) {
#pragma unroll
    for (int j = 0; j < kCols; ++j)
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(park + (uint32_t)(((col0 + j) * kTileR + row_in_tile) * 4)),
                   "f"(acc[j])
                   : "memory");
  }
  __syncwarp();
  cluster_sync_all();
  if (warp < E) {
    if (split == 1)
      finish_rows<E, BN, kFinish, 1>(p, qkv, place, park, rank, tn, tt * BN, warp, lane);
    else if (split == 2)
      finish_rows<E, BN, kFinish, 2>(p, qkv, place, park, rank, tn, tt * BN, warp, lane);
    else if (split == 4)
      finish_rows<E, BN, kFinish, 4>(p, qkv, place, park, rank, tn, tt * BN, warp, lane);
    else if constexpr (!kPairs)
      finish_rows<E, BN, kFinish, 8>(p, qkv, place, park, rank, tn, tt * BN, warp, lane);
  }
  __syncwarp();
  if (gridDim.y > 1) cluster_sync_all();  // no CTA leaves while a peer may still read its rows

  tc_fence_before();
  __syncthreads();
  if (warp == E + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// --------------------------------------------------------------------------
// Wide kernel (more than 128 tokens): tokens are the 128 UMMA rows, 256 weight rows the columns.
//
//   * Schedule, grid = (CTAs, split).  With at least as many tiles as SMs the grid is persistent (split =
//     1, one CTA per SM): CTA c takes tiles c, c + P, c + 2P, ... whole and stores a finished tile while
//     the tensor core already works on the next one.  A shape with fewer tiles than SMs runs one tile per
//     2- or 4-CTA cluster, each CTA taking a slice of K: every CTA parks its fp32 partial in its own (then
//     idle) stage ring in a swizzled [row][4-column group] layout, and after a cluster barrier reads the
//     column slice it owns from every peer with 16-byte distributed-shared-memory loads, adds the partials
//     in rank order (a fixed order: results do not depend on timing) and stores bf16.  No global scratch.
//   * Two 256-column accumulators ping-pong in TMEM, each with its own MMA issuer thread, and a K block has one
//     commit, on the barrier that both frees its stage and hands its accumulator over: one thread's wait, four MMAs
//     and commit take about 770 cycles, the MMAs 512 (two issuers measured 512 with nothing to promote).  An issuer has
//     the operands' barrier behind it and its descriptors at hand when the accumulator comes back.
//   * 20 warps: 16 promotion warps, one TMA producer, two MMA issuers, one idle.  A promotion warp keeps 32 rows x 64
//     columns of the fp32 result in registers and adds a K block in two loads of 32 columns (packed fp32x2
//     multiply-adds); four warps per scheduler hide the loads' latency (eight warps with 128 columns each and the
//     loads pipelined by hand: 4736 x 19456 x 2560 307 us, sixteen 264).  The accumulator goes back to its issuer
//     as soon as the second load has landed.  A thread requests its row's scale one K block ahead, unconditionally (dead
//     rows and columns read scales that nothing is stored from): under a condition the loads were waited for on the spot.
//     With the issuers' order, 560 x 19456 x 2560 43.9 -> 38.9 us, 4736 tokens 256 -> 242, 12032 687 -> 622.
//   * What bounds it now, 4736 x 19456 x 2560 (242 us): 174 us without operand loads and promotion, 212 with the promotion,
//     208 with the loads: MMA operand reads and TMA writes share 128 bytes a clock of shared memory.
//   * A pair of CTAs on one 256 x 256 tile (cta_group::2, a third less operand traffic) measured 3 % faster at 12032
//     tokens and up to 20 % slower at a few hundred, where its tiles leave more rows empty.
// --------------------------------------------------------------------------
constexpr int kWideBN = 256;
constexpr int kWideEpiWarps = 16;
constexpr int kWideThreads = 640;
constexpr int kWideStoreBytes = kWideEpiWarps * 2048;  // per promotion warp: 32 rows x 32 columns of 16-bit output

constexpr int kWideStages = 4;
constexpr int kWideAcc = 2;
constexpr int kWideStageBytes = kTileR * kBlockK + kWideBN * kBlockK;  // 48 KiB
constexpr int kWideSmemBytes =
    kWideStages * kWideStageBytes + kWideStoreBytes + (2 * kWideStages + kWideAcc) * 8 + 64 + 1024;
static_assert(kWideStages * kWideStageBytes >= kTileR * kWideBN * 4, "stage ring too small for the fp32 partial tile");
static_assert(kWideAcc <= kWideStages, "a done barrier must not run a phase ahead of the promotion");

struct WideItem {
  int tm, tn, k0, k1;
};

// Work of CTA (x, rank) of a (gridDim.x, split) grid over the launch's tiles.  split == 1: tiles
// first + x, first + x + gridDim.x, ... whole.  split > 1 (one cluster per tile): tile first + x, the
// rank-th part of its K range.  Tiles are numbered down the token tiles of a band, then along the weight tiles, then band
// by band (band: see wide_band).
__device__ __forceinline__ bool wide_item(const GemmParams& p, int idx, WideItem& it) {
  const int tile = p.tile_begin + (int)blockIdx.x + idx * (int)gridDim.x;
  const int split = gridDim.y, rank = blockIdx.y;
  if (tile >= p.tile_end || (split > 1 && idx > 0)) return false;
  const int tiles_m = (p.m + kTileR - 1) / kTileR, tiles_n = (p.n + kWideBN - 1) / kWideBN;
  const int kb_total = (p.k + kBlockK - 1) / kBlockK;
  const int band = tile / (p.band * tiles_n), in_band = tile - band * p.band * tiles_n;
  const int rows = tiles_m - band * p.band < p.band ? tiles_m - band * p.band : p.band;
  it.tn = in_band / rows;
  it.tm = band * p.band + in_band - it.tn * rows;
  it.k0 = (int)((long long)kb_total * rank / split);
  it.k1 = (int)((long long)kb_total * (rank + 1) / split);
  return true;
}

__device__ __forceinline__ void tmem_ld_wait_pin(float (&a)[32]) {
  // The wait is what makes the registers of the earlier tcgen05.ld valid; naming them as in/out operands
  // keeps every later use of a behind it.
  uint32_t* r = reinterpret_cast<uint32_t*>(a);
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Token tiles per band: all when the activations take less than about a quarter of L2, else equal bands of less.  12032 x
// 2560 x 9728 (117 MB of activations, read again for every column of tiles): 320 us as one band, 284 in bands of 20;
// 4736 x 19456 x 2560 (12 MB): 242 as one, 248 in bands of 20 (fewer CTAs at the same weights).
inline int wide_band(int m, int k) {
  const int tiles_m = (m + kTileR - 1) / kTileR;
  const int bands = (int)(((long long)m * k + (32 << 20) - 1) / (32 << 20));
  return (tiles_m + bands - 1) / bands;
}

// acc[0..32) += d[0..32) * s, two columns per instruction.
__device__ __forceinline__ void promote32(float* acc, const float (&d)[32], float s) {
  const float2 s2 = make_float2(s, s);
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const float2 r = __ffma2_rn(make_float2(d[j], d[j + 1]), s2, make_float2(acc[j], acc[j + 1]));
    acc[j] = r.x;
    acc[j + 1] = r.y;
  }
}

// Cluster reduction of a K-split tile: this CTA adds the 4-column groups [g_lo, g_lo + 64 / kSplit) of the
// tile over all ranks, in rank order, and stores them.  A thread owns 32 / kSplit (row, group) items and has
// the loads of all of them, from every rank, in flight together (one exposed round trip instead of many).
template <int kSplit>
__device__ __forceinline__ void wide_cluster_reduce(const GemmParams& p, uint32_t park_addr, int rank, int epi_tid,
                                                    int tok0, int col_base) {
  constexpr int kGroups = 64 / kSplit, kItems = kTileR * kGroups / (kWideEpiWarps * 32);
  const int g_lo = kGroups * rank;
  const bool vec = (p.ldy % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.y) & 7) == 0);
  float4 part[kItems][kSplit];
#pragma unroll
  for (int u = 0; u < kItems; ++u) {
    const int i = epi_tid + u * (kWideEpiWarps * 32);
    const int row = i / kGroups, g = g_lo + i % kGroups;
    const uint32_t slot = park_addr + (uint32_t)((row * 64 + (g ^ (row & 7))) * 16);
#pragma unroll
    for (int peer = 0; peer < kSplit; ++peer) part[u][peer] = ld_cluster_f4(slot, (uint32_t)peer);
  }
#pragma unroll
  for (int u = 0; u < kItems; ++u) {
    const int i = epi_tid + u * (kWideEpiWarps * 32);
    const int row = i / kGroups, g = g_lo + i % kGroups;
    float4 sum = part[u][0];
#pragma unroll
    for (int peer = 1; peer < kSplit; ++peer) {
      sum.x += part[u][peer].x;
      sum.y += part[u][peer].y;
      sum.z += part[u][peer].z;
      sum.w += part[u][peer].w;
    }
    const int tok = tok0 + row, n0 = col_base + g * 4;
    if (tok < p.m && n0 < p.n) {
      uint16_t* dst = reinterpret_cast<uint16_t*>(p.y) + (long long)tok * p.ldy + n0;
      if (vec && n0 + 4 <= p.n) {
        uint2 w;
        w.x = p.out_f16 ? Mma16816<__half>::pack(sum.x, sum.y) : Mma16816<__nv_bfloat16>::pack(sum.x, sum.y);
        w.y = p.out_f16 ? Mma16816<__half>::pack(sum.z, sum.w) : Mma16816<__nv_bfloat16>::pack(sum.z, sum.w);
        *reinterpret_cast<uint2*>(dst) = w;
      } else {
        const float v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (n0 + j < p.n) {
            if (p.out_f16)
              reinterpret_cast<__half*>(dst)[j] = __float2half_rn(v[j]);
            else
              reinterpret_cast<__nv_bfloat16*>(dst)[j] = __float2bfloat16_rn(v[j]);
          }
        }
      }
    }
  }
}

// Finish::kSilu of the wide kernel: a tile has 128 gate columns and the 128 up columns that belong to them.  Warps w and
// w + 8 have the gate and up values of the same 32 rows and 64 columns; each passes the other half of its columns and
// finishes 32, whose largest value meets those of the row's three other warps.  The staging area holds 64 bytes a row and
// warp: bf16 values for the partner, then, in the place a lane has just read, its maximum.
__device__ __forceinline__ void wide_finish_silu(const GemmParams& p, const WideItem& it, const float (&acc)[64],
                                                 uint8_t* stores, int warp, int lane, bool ok) {
  const int quad = warp & 3, group = warp >> 2;
  const bool gate = group < 2;  // keeps columns [0, 32) of its 64, the up warp [32, 64)
  auto slot = [&](int w, int u) {
    return reinterpret_cast<uint4*>(stores + w * 2048) + lane * 4 + ((u + (lane >> 1)) & 3);
  };
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = u * 8 + 2 * q;
      w[q] = gate ? Mma16816<__nv_bfloat16>::pack(acc[32 + j], acc[33 + j]) : Mma16816<__nv_bfloat16>::pack(acc[j], acc[j + 1]);
    }
    *slot(warp, u) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 7)) : "memory");
  float v[4][8], amax = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    Bf16x8 theirs, mine, r;
    theirs.raw = *slot(warp ^ 8, u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = u * 8 + 2 * q;
      mine.word[q] = gate ? Mma16816<__nv_bfloat16>::pack(acc[j], acc[j + 1]) : Mma16816<__nv_bfloat16>::pack(acc[32 + j], acc[33 + j]);
    }
    // The rounding points of the unfused chain: gate and up to bf16, SiLU to bf16, their product to bf16.
    float g[8];
    unpack8(gate ? mine.raw : theirs.raw, g);
    silu8(g, v[u]);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      r.pair[q] = __hmul2_rn(__floats2bfloat162_rn(v[u][2 * q], v[u][2 * q + 1]), gate ? theirs.pair[q] : mine.pair[q]);
    unpack8(r.raw, v[u]);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[u][j]));
  }
  *reinterpret_cast<float*>(slot(warp ^ 8, 0)) = amax;
  asm volatile("bar.sync %0, 128;" ::"r"(9 + quad) : "memory");
#pragma unroll
  for (int x = 0; x < 4; ++x) amax = fmaxf(amax, *reinterpret_cast<const float*>(slot(x * 4 + quad, 0)));
  asm volatile("bar.sync %0, 128;" ::"r"(9 + quad) : "memory");  // before the next tile's values
  const int row = it.tm * kTileR + quad * 32 + lane;
  if (row >= p.m || !ok) return;
  const float scale = __fdiv_rn(amax, 448.0f), denom = fmaxf(scale, 1e-12f);
  uint8_t* dst = p.q + (long long)row * p.ldq + it.tn * 128 + (group & 1) * 64 + (gate ? 0 : 32);
  const bool wide = ((reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
#pragma unroll
  for (int u = 0; u < 4; u += 2) {
    uint32_t lo[2], hi[2];
    quantize_values(v[u], denom, lo);
    quantize_values(v[u + 1], denom, hi);
    if (wide) {
      *reinterpret_cast<uint4*>(dst + u * 8) = make_uint4(lo[0], lo[1], hi[0], hi[1]);
    } else {
      uint32_t* d = reinterpret_cast<uint32_t*>(dst + u * 8);
      d[0] = lo[0], d[1] = lo[1], d[2] = hi[0], d[3] = hi[1];
    }
  }
  if (group == 0) p.q_scales[(long long)it.tn * p.q_scale_ld + row] = scale;
}

template <Finish kFinish>
__global__ void __launch_bounds__(kWideThreads, 1)
    fp8_gemm_wide_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                         const GemmParams p) {
  constexpr int BN = kWideBN, E = kWideEpiWarps, kStages = kWideStages, kStageBytes = kWideStageBytes;
  constexpr int kAcc = kWideAcc;
  constexpr int kCols = BN * 4 / E;  // columns owned by one promotion warp
  constexpr uint32_t kTmemCols = 512;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* stage_base = smem;
  uint8_t* store_base = smem + kStages * kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(store_base + kWideStoreBytes);
  uint64_t* done_bar = full_bar + kStages;  // the MMAs of the stage's K block have completed
  uint64_t* tmem_empty = done_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + kAcc);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int split = gridDim.y, rank = blockIdx.y;  // cluster = (1, split, 1)

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&done_bar[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) mbar_init(&tmem_empty[b], E);
    mbar_fence_init();
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_w);
  }
  if (warp == E + 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto load_x = [&](uint32_t s, int kb, const WideItem& it) {
    tma_load_2d(stage_base + (size_t)s * kStageBytes, &map_x, &full_bar[s], kb * kBlockK, it.tm * kTileR);
  };
  auto load_w = [&](uint32_t s, int kb, const WideItem& it) {
    uint8_t* dst = stage_base + (size_t)s * kStageBytes + kTileR * kBlockK;
    if constexpr (kFinish == Finish::kSilu) {  // boxes of 128 rows: gate, up
      tma_load_2d(dst, &map_w, &full_bar[s], kb * kBlockK, it.tn * 128);
      tma_load_2d(dst + 128 * kBlockK, &map_w, &full_bar[s], kb * kBlockK, p.n / 2 + it.tn * 128);
    } else {
      tma_load_2d(dst, &map_w, &full_bar[s], kb * kBlockK, it.tn * BN);
    }
  };
  // Barriers, tensor-map prefetch and the TMEM allocation above overlap the tail of the previous kernel.
  // So can static weights (nothing on the stream writes them): the producer requests the weight half of its
  // first stages before the launch-chain wait and adds the activation half afterwards.
  uint32_t prefetched = 0;
  if (p.prefetch && warp == E && lane == 0) {
    WideItem first;
    if (wide_item(p, 0, first)) {
      for (int kb = first.k0; kb < first.k1 && prefetched < (uint32_t)kStages; ++kb, ++prefetched) {
        mbar_expect_tx(&full_bar[prefetched], kStageBytes);
        load_w(prefetched, kb, first);
      }
    }
  }
  if (p.early_release) chain_release();
  if (!p.late_wait) chain_wait();
  if (!p.early_release) chain_release();

  // K blocks this CTA will process (the promotion pipeline needs to know when the last one is reached).
  uint32_t total_blocks = 0;
  {
    WideItem it;
    for (int idx = 0; wide_item(p, idx, it); ++idx)
      total_blocks += (uint32_t)(it.k1 - it.k0);
  }

  if (warp >= E) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == E && lane == 0) {
      // ---------------- TMA producer ----------------
      uint32_t n = 0;
      bool ok = true;
      WideItem it;
      for (int idx = 0; ok && wide_item(p, idx, it); ++idx) {
        for (int kb = it.k0; kb < it.k1; ++kb, ++n) {
          const uint32_t s = n % kStages;
          if (n < prefetched) {  // the weight half is already on its way
            load_x(s, kb, it);
            continue;
          }
          if (!mbar_wait_bounded(&done_bar[s], ((n / kStages) & 1u) ^ 1u)) {
            raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
            ok = false;
            break;
          }
          mbar_expect_tx(&full_bar[s], kStageBytes);
          load_x(s, kb, it);
          load_w(s, kb, it);
        }
      }
    } else if (warp == E + 1 || warp == E + 2) {
      // ---------------- MMA issuers, one per accumulator ----------------
      constexpr uint32_t idesc = instr_desc_f8(BN);
      static_assert(kStages == 2 * kAcc, "issuer b has stages b and b + 2");
      const int b = warp - (E + 1);
      const uint32_t addr = smem_u32(stage_base + (size_t)b * kStageBytes), tmem_d = tmem_base + b * BN;
      const uint64_t da0 = smem_desc_k128(addr), db0 = smem_desc_k128(addr + kTileR * kBlockK);
      uint32_t second = 0, parity = 0;  // stage b or b + kAcc, phase of that stage
#pragma unroll 1
      for (uint32_t n = b; n < total_blocks; n += kAcc) {
        const uint64_t da = da0 + second * (kAcc * kStageBytes >> 4), db = db0 + second * (kAcc * kStageBytes >> 4);
        uint64_t* done = &done_bar[b + second * kAcc];
        if (!warp_wait_bounded(&full_bar[b + second * kAcc], parity) ||
            !warp_wait_bounded(&tmem_empty[b], second ^ 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          break;
        }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k)
            umma_f8(tmem_d, da + (uint64_t)(k * kUmmaK / 16), db + (uint64_t)(k * kUmmaK / 16), idesc, k > 0 ? 1u : 0u);
          umma_commit(done);  // frees the smem stage and hands the accumulator to the promotion warps
        }
        __syncwarp();
        parity ^= second;
        second ^= 1u;
      }
    }
    __syncwarp();
    if (split > 1) {
      cluster_sync_all();  // partials parked
      cluster_sync_all();  // peers have read this CTA's partial
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // ---------------- Promotion warps ----------------
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    const int col0 = (warp >> 2) * kCols;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)col0;
    const int epi_tid = threadIdx.x;
    float acc[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    uint32_t n = 0;
    bool ok = true;
    WideItem it;
    // A failed wait only clears `ok` where warps meet at the end of a tile: all of them pass the same barriers.
    constexpr bool kMeet = kFinish == Finish::kSilu;
    for (int idx = 0; (ok || kMeet) && wide_item(p, idx, it); ++idx) {
      const int tok0 = it.tm * kTileR;
      // The scales of this thread's row and of its columns' weight block, requested a K block ahead.  Ordinary loads: the
      // kernel before may have written them while this one was waiting, which the read-only path does not allow for.
      const int blk = kFinish == Finish::kSilu ? it.tn + (col0 / 128) * (p.n / 256) : it.tn * 2 + col0 / 128;
      const bool row_live = tok0 + row_in_tile < p.m, col_live = blk * 128 < p.n;
      const float* a_at = p.a_scale + (long long)it.k0 * p.a_scale_ld + (row_live ? tok0 + row_in_tile : 0);
      const float* w_at = p.w_scale + (col_live ? (long long)blk * p.w_scale_ld : 0) + it.k0;
      float a_next = *a_at, w_next = *w_at;
      for (int kb = it.k0; (ok || !kMeet) && kb < it.k1; ++kb, ++n) {
        const uint32_t taddr = lane_addr + (n & 1) * BN;
        if (!mbar_wait_bounded(&done_bar[n % kStages], (n / kStages) & 1u)) {
          raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
          ok = false;
          break;
        }
        tc_fence_after();
        const float s = a_next * w_next;
        a_at += kb + 1 < it.k1 ? p.a_scale_ld : 0;
        w_at += kb + 1 < it.k1 ? 1 : 0;
        a_next = *a_at;
        w_next = *w_at;
        float buf[32];
        tmem_ld32(taddr, buf);
        tmem_ld_wait_pin(buf);
        promote32(acc, buf, s);
        tmem_ld32(taddr + 32, buf);
        tmem_ld_wait_pin(buf);
        // Every load of this accumulator has landed: hand the buffer back to the MMA issuer.
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[n & 1]);
        promote32(acc + 32, buf, s);
      }
      if (!ok && !kMeet) break;

      const int r_glob = tok0 + row_in_tile;
      if constexpr (kFinish == Finish::kSilu) {
        wide_finish_silu(p, it, acc, store_base, warp, lane, ok);
      } else if (split == 1) {
        const int n0 = it.tn * BN + col0;
        const bool vec = (p.ldy % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.y) & 15) == 0) && (n0 + kCols <= p.n);
        if (vec) {
          // Rows leave through a per-warp staging area so that global stores are whole 64-byte row
          // segments: a lane parks 32 columns of its own row (4 x 16 bytes, unit u of row r at
          // r * 4 + ((u + r / 2) & 3): conflict-free both ways), then four lanes store one row segment.
          uint4* stage = reinterpret_cast<uint4*>(store_base + warp * 2048);
          const int out_row = lane >> 2, unit = lane & 3;
#pragma unroll
          for (int c = 0; c < kCols; c += 32) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint32_t w[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int j = c + u * 8 + 2 * q;
                w[q] = p.out_f16 ? Mma16816<__half>::pack(acc[j], acc[j + 1])
                                 : Mma16816<__nv_bfloat16>::pack(acc[j], acc[j + 1]);
              }
              stage[lane * 4 + ((u + (lane >> 1)) & 3)] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            __syncwarp();
#pragma unroll
            for (int r8 = 0; r8 < 32; r8 += 8) {
              const int r = r8 + out_row;
              const uint4 v = stage[r * 4 + ((unit + (r >> 1)) & 3)];
              const int tok = tok0 + quad * 32 + r;
              if (tok < p.m) {
                uint16_t* dst = reinterpret_cast<uint16_t*>(p.y) + (long long)tok * p.ldy + n0 + c + unit * 8;
                *reinterpret_cast<uint4*>(dst) = v;
              }
            }
            __syncwarp();
          }
        } else if (r_glob < p.m) {
          uint16_t* yrow = reinterpret_cast<uint16_t*>(p.y) + (long long)r_glob * p.ldy + n0;
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            if (n0 + j < p.n) {
              if (p.out_f16)
                reinterpret_cast<__half*>(yrow)[j] = __float2half_rn(acc[j]);
              else
                reinterpret_cast<__nv_bfloat16*>(yrow)[j] = __float2bfloat16_rn(acc[j]);
            }
          }
        }
      } else {
        // Park the partial: float4 (row, g) lives at slot row * 64 + (g ^ (row & 7)), so that both the
        // row-per-lane writes here and the column-group-per-lane reads below are free of bank conflicts.
        // Every MMA of this CTA has completed (its last accumulator was consumed), so the ring is idle.
        float4* park = reinterpret_cast<float4*>(stage_base);
#pragma unroll
        for (int j = 0; j < kCols; j += 4) {
          const int g = (col0 + j) >> 2;
          park[row_in_tile * 64 + (g ^ (row_in_tile & 7))] = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
        cluster_sync_all();
        if (split == 2)
          wide_cluster_reduce<2>(p, smem_u32(stage_base), rank, epi_tid, tok0, it.tn * BN);
        else
          wide_cluster_reduce<4>(p, smem_u32(stage_base), rank, epi_tid, tok0, it.tn * BN);
        cluster_sync_all();  // no CTA leaves while a peer may still read its partial
      }
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    }
    if (!ok) {
      tmem_ld_wait();  // nothing of this thread stays in flight
      if (split > 1) {  // a CTA that gave up still meets its peers at the two cluster barriers
        cluster_sync_all();
        cluster_sync_all();
      }
    }
  }

  // Second launch of a two-launch GEMM: it ran beside the first one, and must not complete before it
  // (the kernel queued behind only waits for this one).
  if (p.late_wait) chain_wait();
  tc_fence_before();
  __syncthreads();
  if (warp == E + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// --------------------------------------------------------------------------
// Activation quantiser: per token, per 128 columns.  One half-warp per group, eight columns a lane.  Bound by HBM (3
// bytes a value) with the quotients by corrected_quotient and 32-bit indices; with IEEE divisions and a 64-bit index
// division it was bound by instructions (12032 x 4096: 52.4 us, now 39.7 us).
// --------------------------------------------------------------------------
template <typename T, typename Index>
__global__ void quantize_kernel(const T* x, long long ldx, uint8_t* q, long long ldq, float* scales, int scale_ld,
                                int m, int k) {
  chain_release();
  chain_wait();
  const Index groups = (Index)((k + 127) / 128);
  const Index hw = ((Index)blockIdx.x * (Index)blockDim.x + threadIdx.x) >> 4;  // half-warp id
  const int l16 = threadIdx.x & 15;
  const bool live = hw < (Index)m * groups;  // dead lanes still take part in the shuffles
  const int row = live ? (int)(hw / groups) : 0, grp = live ? (int)(hw - (Index)row * groups) : 0;
  const int c0 = grp * 128 + l16 * 8;
  float v[8];
  const T* src = x + (long long)row * ldx + c0;
  if (!live) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
  } else if (c0 + 8 <= k && ((reinterpret_cast<uintptr_t>(src) & 15) == 0)) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = to_float<T>(e[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = c0 + j < k ? to_float<T>(src[j]) : 0.f;
  }
  uint32_t packed[2];
  float scale;  // the raw scale is what gets stored (0 for a zero group)
  quantize_group(v, packed, scale);
  if (!live) return;
  uint8_t* dst = q + (long long)row * ldq + c0;
  if (c0 + 8 <= k && ((reinterpret_cast<uintptr_t>(dst) & 7) == 0)) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
  } else {
    const uint8_t* b = reinterpret_cast<const uint8_t*>(packed);
    for (int j = 0; j < 8; ++j)
      if (c0 + j < k) dst[j] = b[j];
  }
  if (l16 == 0) scales[(long long)grp * scale_ld + row] = scale;
}

template <typename T>
int launch_quantize(const void* x, long long ldx, void* q, long long ldq, float* scales, int scale_ld, int m, int k,
                    cudaStream_t stream) {
  const int threads = 256;
  const long long half_warps = (long long)m * ((k + 127) / 128), blocks = (half_warps * 16 + threads - 1) / threads;
  const dim3 grid((unsigned)blocks), block(threads);
  if (blocks * threads < (1ll << 31))
    MIE_CUDA(launch_chained(quantize_kernel<T, uint32_t>, grid, block, 0, stream, (const T*)x, ldx, (uint8_t*)q, ldq,
                            scales, scale_ld, m, k));
  else
    MIE_CUDA(launch_chained(quantize_kernel<T, uint64_t>, grid, block, 0, stream, (const T*)x, ldx, (uint8_t*)q, ldq,
                            scales, scale_ld, m, k));
  MIE_LAUNCH_CHECK("quantize_kernel");
  return MIE_OK;
}

// --------------------------------------------------------------------------
// Host side
// --------------------------------------------------------------------------
struct Map2Key {
  const void* ptr;
  long long rows, k, ld;
  int box_rows;
  bool operator==(const Map2Key& o) const {
    return ptr == o.ptr && rows == o.rows && k == o.k && ld == o.ld && box_rows == o.box_rows;
  }
};
struct Map2Hash {
  size_t operator()(const Map2Key& k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr);
    h = h * 1000003u ^ (size_t)k.rows;
    h = h * 1000003u ^ (size_t)k.k;
    h = h * 1000003u ^ (size_t)k.ld;
    h = h * 1000003u ^ (size_t)k.box_rows;
    return h;
  }
};

int operand_map(const void* ptr, long long rows, long long k, long long ld, int box_rows, CUtensorMap* out) {
  static std::mutex mu;
  static std::unordered_map<Map2Key, CUtensorMap, Map2Hash> cache;
  Map2Key key{ptr, rows, k, ld, box_rows};
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return MIE_OK;
    }
  }
  const uint64_t dims[2] = {(uint64_t)k, (uint64_t)rows};
  const uint64_t strides[1] = {(uint64_t)ld};
  const uint32_t box[2] = {(uint32_t)kBlockK, (uint32_t)box_rows};
  const int rc = make_tensor_map(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box,
                                 CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != MIE_OK) return rc;
  std::lock_guard<std::mutex> lock(mu);
  if (cache.size() > 16384) cache.clear();
  cache.emplace(key, *out);
  return MIE_OK;
}

// K-split factor for a shape with `tiles` output tiles of `kb_total` K blocks.  Cost model in units of
// one K block of a 256-column tile: waves * (K blocks per CTA + fixed cost) + the cluster reduction
// (which grows with the tile width).  Cluster sizes 1, 2 and 4 are used, and 8 for the narrow tiles that
// run two 100 KB CTAs per SM (o / down at up to 32 tokens: 160 CTAs instead of 80); 3 and 8 co-schedule
// badly with one 200 KB CTA per SM (measured), and larger splits leave too little work per CTA.
int choose_split(long long tiles, int kb_total, int bn, int ctas_per_sm, int max_split, int limit) {
  const int slots = sm_count() * ctas_per_sm;
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= limit; s *= 2) {
    if (s > kb_total || (max_split > 0 && s > max_split)) break;
    const long long ctas = tiles * s;
    const double waves = (double)((ctas + slots - 1) / slots);
    const double cost = waves * ((kb_total + s - 1) / s + 4.0) + (s > 1 ? bn / 32.0 : 0.0);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

template <int BN, Finish kFinish, int E>
int launch_narrow_tiles(const CUtensorMap& mw, const CUtensorMap& mx, const GemmParams& p, const QkvParams& qkv,
                        int tiles, int split, cudaStream_t stream) {
  using S = GemmSmem<BN>;
  static bool configured[64] = {false};
  int dev = 0;
  MIE_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    MIE_CUDA(cudaFuncSetAttribute(fp8_gemm_kernel<BN, kFinish, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  S::kTotal));
    configured[dev] = true;
  }
  constexpr int kPair = kFinish == Finish::kSilu ? 2 : 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(tiles / kPair), (unsigned)(split * kPair), 1);
  config.blockDim = dim3(narrow_threads(E), 1, 1);
  config.dynamicSmemBytes = S::kTotal;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = (unsigned)(split * kPair);
  attr[0].val.clusterDim.z = 1;
  config.attrs = attr;
  config.numAttrs = chained_launch_enabled() ? 2 : 1;
  MIE_CUDA(cudaLaunchKernelEx(&config, fp8_gemm_kernel<BN, kFinish, E>, mw, mx, p, qkv));
  MIE_LAUNCH_CHECK("fp8_gemm_kernel");
  return MIE_OK;
}

template <int BN, Finish kFinish>
int launch_narrow_columns(const CUtensorMap& mw, const CUtensorMap& mx, const GemmParams& p, const QkvParams& qkv,
                          int max_split, cudaStream_t stream) {
  constexpr int kPerSm = GemmSmem<BN>::kCtasPerSm, kPair = kFinish == Finish::kSilu ? 2 : 1;
  const long long tiles = (long long)((p.n + kTileR - 1) / kTileR) * ((p.m + BN - 1) / BN);
  MIE_CHECK_ARG(tiles <= 0x7fffffff, "too many output tiles (%lld)", tiles);
  const int kb = (p.k + kBlockK - 1) / kBlockK;
  const int split = choose_split(tiles, kb, BN, kPerSm, max_split, (kPerSm == 2 ? 8 : 4) / kPair);
  constexpr int kFew = narrow_warps(BN, 1), kMany = narrow_warps(BN, 1 << 20);
  if (narrow_warps(BN, (kb + split - 1) / split) == kFew)
    return launch_narrow_tiles<BN, kFinish, kFew>(mw, mx, p, qkv, (int)tiles, split, stream);
  return launch_narrow_tiles<BN, kFinish, kMany>(mw, mx, p, qkv, (int)tiles, split, stream);
}

// Column-tile width for the swapped orientation: smallest of 16/32/64/128 covering m.
int swap_bn(int m) { return m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128; }

template <Finish kFinish>
int launch_narrow(const void* x8, long long ldx, const void* w8, long long ldw, const GemmParams& p,
                  const QkvParams& qkv, int max_split, cudaStream_t stream) {
  const int bn = swap_bn(p.m);
  CUtensorMap mw, mx;
  if (int rc = operand_map(w8, p.n, p.k, ldw, kTileR, &mw)) return rc;
  if (int rc = operand_map(x8, p.m, p.k, ldx, bn, &mx)) return rc;
  switch (bn) {
    case 16: return launch_narrow_columns<16, kFinish>(mw, mx, p, qkv, max_split, stream);
    case 32: return launch_narrow_columns<32, kFinish>(mw, mx, p, qkv, max_split, stream);
    case 64: return launch_narrow_columns<64, kFinish>(mw, mx, p, qkv, max_split, stream);
    default: return launch_narrow_columns<128, kFinish>(mw, mx, p, qkv, max_split, stream);
  }
}

// Whether m tokens of an n-row weight take the narrow kernel: up to 128 tokens, unless that needs a second wave (more
// 128-row weight tiles than SMs at more than 32 tokens, where only one of its CTAs fits an SM: gate_up): the wide
// kernel's 256-row tiles then finish in one round.
bool narrow_fits(int m, int n) {
  return m <= 32 || (m <= 128 && (n + kTileR - 1) / kTileR <= sm_count());
}

// Whether finishing the rows in the projection beats storing them for a second kernel.  It saves about 1.1 us of launch and
// reading, but a CTA finishes its share of the tokens alone, and gate and up rows of a tile take two CTAs of the cluster,
// which leaves K half as many parts.  Measured (us, separate / finished):
//   q/k/v   up to 32 tokens everywhere (1 token of 6144 x 2560 8.6 / 7.3); then only with K cut, so that several CTAs share
//           the tokens: 64 tokens of 3072 x 2560 in 2 parts or more 10.4 / 8.6, of 6144 x 512 uncut 8.6 / 10.4; 128 tokens
//           of 1536 x 2560 in 4 parts 11.8 / 11.4, of 6144 x 4096 in 2 18.9 / 19.7.
//   gated   up to 32 tokens (1 token of 9728 x 2560 10.1 / 8.8, of 19456 x 2560 13.1 / 12.7) unless the halved split shows
//           (1024 x 8192 7.5 / 8.0) or its clusters of four nearly fill the GPU and not all find room at once (18688 x 4096
//           16.9 / 22.1); then with K cut into as many parts as without (64 tokens of 6144 x 4096 12.6 / 11.6, of
//           2048 x 4096 9.5 / 10.5) or, up to 64 tokens, short (1536 x 1024 7.5 / 6.9); above 64 not of a short uncut K
//           (1024 x 512 8.5 / 10.7; 12288 x 2048 19.0 / 18.1).
bool finish_pays(int m, int n, int k, bool gated, int max_split) {
  if (!narrow_fits(m, n)) return false;
  const int bn = swap_bn(m), per_sm = m <= 32 ? 2 : 1, limit = m <= 32 ? 8 : 4;
  const int tiles = (n + kTileR - 1) / kTileR, kb = (k + kBlockK - 1) / kBlockK;
  const int stored = choose_split(tiles, kb, bn, per_sm, max_split, limit);
  if (!gated) return m <= 32 || stored >= (m <= 64 ? 2 : 4);
  const int split = choose_split(tiles, kb, bn, per_sm, max_split, limit / 2);
  if (split > 1 && tiles * split > per_sm * sm_count() * 9 / 10) return false;
  if (m <= 32) return split == stored || kb < 64;
  if (m <= 64) return split == stored || kb <= 8;
  return split == stored && (split > 1 || kb >= 16);
}

// Schedule of the wide kernel.  `tiles` output tiles of `kb` K blocks on P SMs (one 200 KB CTA each):
//   tiles <= P      one launch; whole tiles, or one tile per 2-/4-CTA cluster with the K range cut when all
//                   clusters still fit one wave;
//   tiles > P       the whole waves (floor(tiles / P) * P tiles) run as one persistent launch; the
//                   remaining R tiles would otherwise cost a full extra round on R of the P SMs, so when
//                   R * s <= P they go to a second launch of one s-CTA cluster per tile (s = 2 or 4) that
//                   starts on the SMs the first launch frees and finishes in 1 / s of a round.
// Costs in units of one K block of the main loop; the cluster reduction and the fill / drain of a CTA are
// worth a few blocks each.
struct WidePlan {
  int main_tiles;  // tiles of the persistent launch (0: none)
  int main_split;  // K split of the main launch (> 1 only when it is the only launch)
  int tail_split;  // K split of the tail launch (0: no tail launch)
};

WidePlan plan_wide(long long tiles, int kb, int max_split) {
  const int slots = sm_count();
  WidePlan plan{(int)tiles, 1, 0};
  if (tiles <= slots) {
    double best_cost = 1e30;
    for (int s = 1; s <= 4; s *= 2) {
      if (s > kb || (max_split > 0 && s > max_split)) break;
      if (s > 1 && tiles * s > slots) break;  // clusters only when all of them run in one wave
      const double cost = (double)((kb + s - 1) / s) + 4.0 + (s > 1 ? 3.0 : 0.0);
      if (cost < best_cost - 1e-9) {
        best_cost = cost;
        plan.main_split = s;
      }
    }
    return plan;
  }
  const long long rest = tiles % slots;
  if (rest == 0) return plan;
  double best_cost = (double)kb;  // the tail as one more whole round of the persistent launch
  for (int s = 2; s <= 4; s *= 2) {
    if (s > kb || (max_split > 0 && s > max_split) || rest * s > slots) break;
    const double cost = (double)((kb + s - 1) / s) + 3.0 + 2.0;  // reduction + the second launch's start-up
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      plan.main_tiles = (int)(tiles - rest);
      plan.tail_split = s;
    }
  }
  return plan;
}

int launch_wide_range(const CUtensorMap& mx, const CUtensorMap& mw, GemmParams p, int tile_begin, int tile_end,
                      int split, bool late_wait, bool tail_follows, cudaStream_t stream) {
  const auto kernel = p.q != nullptr ? fp8_gemm_wide_kernel<Finish::kSilu> : fp8_gemm_wide_kernel<Finish::kStore>;
  p.tile_begin = tile_begin;
  p.band = wide_band(p.m, p.k);
  p.tile_end = tile_end;
  p.late_wait = late_wait ? 1 : 0;
  p.early_release = tail_follows ? 0 : 1;
  const int count = tile_end - tile_begin;
  const int ctas = split > 1 ? count : (count < sm_count() ? count : sm_count());
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)ctas, (unsigned)split, 1);
  config.blockDim = dim3(kWideThreads, 1, 1);
  config.dynamicSmemBytes = kWideSmemBytes;
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
  MIE_CUDA(cudaLaunchKernelEx(&config, kernel, mx, mw, p));
  MIE_LAUNCH_CHECK("fp8_gemm_wide_kernel");
  return MIE_OK;
}

int launch_wide(const CUtensorMap& mx, const CUtensorMap& mw, const GemmParams& p, int max_split,
                cudaStream_t stream) {
  static bool configured[64] = {false};
  int dev = 0;
  MIE_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    for (const void* kernel : {reinterpret_cast<const void*>(fp8_gemm_wide_kernel<Finish::kStore>),
                               reinterpret_cast<const void*>(fp8_gemm_wide_kernel<Finish::kSilu>)})
      MIE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmemBytes));
    configured[dev] = true;
  }
  const int kb = (p.k + kBlockK - 1) / kBlockK;
  const long long tiles = (long long)((p.m + kTileR - 1) / kTileR) * ((p.n + kWideBN - 1) / kWideBN);
  MIE_CHECK_ARG(tiles <= 0x7fffffff, "too many output tiles (%lld)", tiles);
  if (p.q != nullptr) return launch_wide_range(mx, mw, p, 0, (int)tiles, 1, false, false, stream);  // whole tiles only
  const WidePlan plan = plan_wide(tiles, kb, max_split);
  if (int rc = launch_wide_range(mx, mw, p, 0, plan.main_tiles, plan.main_split, false, plan.tail_split > 0, stream)) return rc;
  if (plan.tail_split > 0) {
    // Only with launch chaining on does the tail start before the main launch has drained; without it the
    // stream simply runs the two launches one after the other.
    return launch_wide_range(mx, mw, p, plan.main_tiles, (int)tiles, plan.tail_split, chained_launch_enabled(),
                             false, stream);
  }
  return MIE_OK;
}

}  // namespace
}  // namespace mie

using namespace mie;

extern "C" int mie_fp8_quantize(const void* x, int64_t ldx, int32_t dtype, void* q, int64_t ldq, float* scales,
                                int32_t scale_ld, int32_t m, int32_t k, void* stream) {
  MIE_CHECK_ARG(x && q && scales, "null pointer");
  MIE_CHECK_ARG(dtype == MIE_DTYPE_BF16 || dtype == MIE_DTYPE_F16, "activation must be bf16 or fp16");
  MIE_CHECK_ARG(m >= 0 && k >= 1 && scale_ld >= m && ldx >= k && ldq >= k, "invalid quantiser shape");
  if (m == 0) return MIE_OK;
  if (dtype == MIE_DTYPE_BF16)
    return launch_quantize<__nv_bfloat16>(x, ldx, q, ldq, scales, scale_ld, m, k, (cudaStream_t)stream);
  return launch_quantize<__half>(x, ldx, q, ldq, scales, scale_ld, m, k, (cudaStream_t)stream);
}

namespace mie {
namespace {

// Argument checks and parameters that the GEMM entry points share.
int gemm_params(GemmParams& p, const void* x8, int64_t ldx, const float* a_scale, int32_t a_scale_ld, const void* w8,
                int64_t ldw, const float* w_scale, int32_t w_scale_ld, int32_t m, int32_t n, int32_t k, int32_t flags,
                int32_t* status) {
  MIE_CHECK_ARG(x8 && a_scale && w8 && w_scale, "null pointer");
  MIE_CHECK_ARG(m >= 0 && n >= 1 && k >= 1, "invalid GEMM shape %d x %d x %d", m, n, k);
  MIE_CHECK_ARG(ldx % 16 == 0 && ldw % 16 == 0, "operand row strides must be multiples of 16 bytes");
  MIE_CHECK_ARG(((reinterpret_cast<uintptr_t>(x8) | reinterpret_cast<uintptr_t>(w8)) & 15) == 0,
                "operands must be 16-byte aligned");
  MIE_CHECK_ARG(a_scale_ld >= m && w_scale_ld >= (k + 127) / 128, "invalid leading dimension");
  MIE_CHECK_ARG((flags & ~(MIE_GEMM_NO_WEIGHT_PREFETCH | MIE_GEMM_STATIC_WEIGHTS)) == 0, "unknown flag bits %d", flags);
  p = GemmParams{};
  p.m = m;
  p.n = n;
  p.k = k;
  p.a_scale = a_scale;
  p.a_scale_ld = a_scale_ld;
  p.w_scale = w_scale;
  p.w_scale_ld = w_scale_ld;
  p.status = status;
  p.prefetch = weight_prefetch_enabled() && flags == MIE_GEMM_STATIC_WEIGHTS;
  return MIE_OK;
}

}  // namespace
}  // namespace mie

extern "C" int mie_fp8_gemm(const void* x8, int64_t ldx, const float* a_scale, int32_t a_scale_ld, const void* w8,
                            int64_t ldw, const float* w_scale, int32_t w_scale_ld, void* y, int64_t ldy,
                            int32_t out_dtype, int32_t m, int32_t n, int32_t k, int32_t max_split, int32_t flags,
                            int32_t* status, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  GemmParams p;
  if (int rc = gemm_params(p, x8, ldx, a_scale, a_scale_ld, w8, ldw, w_scale, w_scale_ld, m, n, k, flags, status))
    return rc;
  MIE_CHECK_ARG(y, "null pointer");
  MIE_CHECK_ARG(out_dtype == MIE_DTYPE_BF16 || out_dtype == MIE_DTYPE_F16, "output must be bf16 or fp16");
  MIE_CHECK_ARG(ldy >= n, "invalid leading dimension");
  if (m == 0) return MIE_OK;
  p.y = y;
  p.ldy = ldy;
  p.out_f16 = out_dtype == MIE_DTYPE_F16;

  // Between 129 and 256 tokens a weight of at most 12 row tiles (N <= 1536: the merged qkv of a 4- or 8-way head shard)
  // is still faster in the narrow kernel, as two token tiles (measured 9.7 vs 12.6 us at N = 768, 10.8 vs 13.1 at
  // N = 1536; at N = 2560 the wide kernel wins).
  if (narrow_fits(m, n) || (m <= 256 && (n + kTileR - 1) / kTileR <= 12))
    return launch_narrow<Finish::kStore>(x8, ldx, w8, ldw, p, QkvParams{}, max_split, stream);
  CUtensorMap mw, mx;
  if (int rc = operand_map(x8, m, k, ldx, kTileR, &mx)) return rc;
  if (int rc = operand_map(w8, n, k, ldw, kWideBN, &mw)) return rc;
  return launch_wide(mx, mw, p, max_split, stream);
}

extern "C" int mie_fp8_gemm_finishes(int32_t m, int32_t n) { return m >= 1 && n >= 1 && narrow_fits(m, n) ? 1 : 0; }

extern "C" int mie_fp8_gemm_finish_pays(int32_t m, int32_t n, int32_t k, int32_t gated, int32_t max_split) {
  return m >= 1 && n >= 1 && k >= 1 && finish_pays(m, n, k, gated != 0, max_split) ? 1 : 0;
}

// Whether the wide kernel should finish the gated rows itself.  It saves a launch and the rows' way through memory, but the
// tensor core has two K blocks to go on with while a tile is finished (about 3 us), and a tail of tiles is not cut.  Measured
// (us, separate / finished), weights [gate | up] of 9728 columns each, K 2560: 300 tokens 32.8 / 32.3, 1024 71.7 / 70.4, 4096
// 257.5 / 242.2, 12032 829 / 812; of 12288, K 4096, 768 tokens 88.8 / 85.8, 12032 1545 / 1527.  What a cut tail is worth grows
// with K and is set against the rounds' gain, about a fifth of a K block each: with K 2560 one round before it is too few (200
// tokens 30.5 / 31.3) and two are enough (400 44.9 / 43.7), with K 3072 three are not (768 63.3 / 63.9) and six are (1536
// 114.2 / 111.4), with K 4096 four are not (1024 95.7 / 96.7) and eight are (2048 180.4 / 174.2).
static bool wide_silu_pays(int m, int cols, int k, int max_split) {
  const long long tiles = (long long)((m + kTileR - 1) / kTileR) * (cols / 128);
  const int kb = (k + kBlockK - 1) / kBlockK;
  if (cols % 128 != 0 || narrow_fits(m, 2 * cols) || tiles > 0x7fffffff) return false;
  const WidePlan plan = plan_wide(tiles, kb, max_split);
  if (plan.main_split > 1) return false;
  const int rounds = plan.main_tiles / sm_count();
  return plan.tail_split == 0 || (kb <= 20 ? rounds >= 2 : 5 * rounds >= kb);
}

extern "C" int mie_fp8_gemm_silu_wide_pays(int32_t m, int32_t cols, int32_t k, int32_t max_split) {
  return m >= 1 && cols >= 1 && k >= 1 && wide_silu_pays(m, cols, k, max_split) ? 1 : 0;
}

extern "C" int mie_fp8_gemm_silu_wide(const void* x8, int64_t ldx, const float* a_scale, int32_t a_scale_ld,
                                      const void* w8, int64_t ldw, const float* w_scale, int32_t w_scale_ld, void* q,
                                      int64_t ldq, float* scales, int32_t scale_ld, int32_t m, int32_t cols, int32_t k,
                                      int32_t flags, int32_t* status, void* stream) {
  MIE_CHECK_ARG(q && scales, "null pointer");
  MIE_CHECK_ARG(cols >= 128 && cols % 128 == 0 && cols <= 0x3fffffff, "cols must be a multiple of 128");
  GemmParams p;
  if (int rc = gemm_params(p, x8, ldx, a_scale, a_scale_ld, w8, ldw, w_scale, w_scale_ld, m, 2 * cols, k, flags, status))
    return rc;
  MIE_CHECK_ARG(scale_ld >= m && ldq >= cols && ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0,
                "the quantised rows must be 4-byte aligned and have scale storage");
  if (m == 0) return MIE_OK;
  p.q = (uint8_t*)q;
  p.ldq = ldq;
  p.q_scales = scales;
  p.q_scale_ld = scale_ld;
  CUtensorMap mw, mx;
  if (int rc = operand_map(x8, m, k, ldx, kTileR, &mx)) return rc;
  if (int rc = operand_map(w8, 2 * cols, k, ldw, 128, &mw)) return rc;
  return launch_wide(mx, mw, p, 1, (cudaStream_t)stream);
}

extern "C" int mie_fp8_gemm_silu(const void* x8, int64_t ldx, const float* a_scale, int32_t a_scale_ld, const void* w8,
                                 int64_t ldw, const float* w_scale, int32_t w_scale_ld, void* q, int64_t ldq,
                                 float* scales, int32_t scale_ld, int32_t m, int32_t cols, int32_t k,
                                 int32_t max_split, int32_t flags, int32_t* status, void* stream) {
  MIE_CHECK_ARG(q && scales, "null pointer");
  MIE_CHECK_ARG(cols >= 128 && cols % 128 == 0 && cols <= 0x3fffffff, "cols must be a multiple of 128");
  GemmParams p;
  if (int rc = gemm_params(p, x8, ldx, a_scale, a_scale_ld, w8, ldw, w_scale, w_scale_ld, m, 2 * cols, k, flags, status))
    return rc;
  MIE_CHECK_ARG(scale_ld >= m && ldq >= cols && ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0,
                "the quantised rows must be 4-byte aligned and have scale storage");
  if (m == 0) return MIE_OK;
  MIE_CHECK_ARG(narrow_fits(m, 2 * cols), "%d tokens of %d columns are not finished in the projection", m, cols);
  p.q = (uint8_t*)q;
  p.ldq = ldq;
  p.q_scales = scales;
  p.q_scale_ld = scale_ld;
  return launch_narrow<Finish::kSilu>(x8, ldx, w8, ldw, p, QkvParams{}, max_split, (cudaStream_t)stream);
}

extern "C" int mie_fp8_gemm_qkv(const void* x8, int64_t ldx, const float* a_scale, int32_t a_scale_ld, const void* w8,
                                int64_t ldw, const float* w_scale, int32_t w_scale_ld, const void* q_weight,
                                const void* k_weight, const void* cos_sin, int32_t max_pos, mie_index_t positions,
                                mie_index_t token_to_sequence, mie_index_t block_tables, void* q_out,
                                mie_view4_t key_blocks, mie_view4_t value_blocks, void* kv_pool,
                                int64_t page_stride_bytes, float* kv_scales, int32_t m, int32_t k, int32_t q_heads,
                                int32_t kv_heads, int32_t block_size, int32_t num_blocks, int32_t table_rows,
                                int32_t table_width, float eps, int32_t max_split, int32_t flags, int32_t* status,
                                void* stream) {
  QkvParams qkv;
  if (int rc = kv_pool != nullptr ? qkv_e4m3_pool(qkv, kv_pool, page_stride_bytes, kv_scales, kv_heads)
                                  : qkv_bf16_pages(qkv, key_blocks, value_blocks))
    return rc;
  MIE_CHECK_ARG(kv_pool == nullptr || block_size == 16, "the e4m3 pool has pages of 16 tokens");
  if (int rc = qkv_common(qkv, q_weight, k_weight, cos_sin, max_pos, positions, token_to_sequence, block_tables, q_out,
                          m, q_heads, kv_heads, block_size, num_blocks, table_rows, table_width, eps, status))
    return rc;
  const long long heads = (long long)q_heads + 2ll * kv_heads;
  MIE_CHECK_ARG(heads <= 0xffffff, "too many heads");
  GemmParams p;
  if (int rc = gemm_params(p, x8, ldx, a_scale, a_scale_ld, w8, ldw, w_scale, w_scale_ld, m, (int)heads * kTileR, k, flags,
                           status))
    return rc;
  if (m == 0) return MIE_OK;
  MIE_CHECK_ARG(narrow_fits(m, p.n), "%d tokens of %lld heads are not finished in the projection", m, heads);
  return launch_narrow<Finish::kQkv>(x8, ldx, w8, ldw, p, qkv, max_split, (cudaStream_t)stream);
}
