// The tcgen05 chunked-prefill attention kernel, shared by the plain entry point (prefill_attention_umma.cu) and
// the one with sinks, windows and other head sizes (sink_prefill_attention.cu).
//
// One CTA = two 128-row query tiles: each 128 / G consecutive query tokens of one request times the G query
// heads that share one KV head, so a K/V tile staged once serves the whole GQA group of both.  Per 128-token K/V
// tile and query tile:
//   S = Q K^T      UMMA 128x128x16 (bf16/fp16, fp32 accumulate), Q and K in shared memory;
//   softmax        a warpgroup per query tile, one thread per row: reads S from TMEM, applies the causal /
//                  length mask and an exp2 softmax against a running reference maximum, and writes
//                  P (16-bit, two per column) back into TMEM over the S it just read;
//   O += P V       UMMA 128x128x16 with P as the TMEM A operand and V as the MN-major shared-memory B
//                  operand, accumulated in TMEM over all tiles.
// The two query tiles take turns: while one's S is on the special-function units the other's products are on the
// tensor core.  TMEM holds S/P and O of both, all 512 columns.
// What bounds it: of 3,040 clocks per K/V tile and pair the products take 2,060 and the exponentials 2,048; a tile's own
// chain is S -> softmax (1,800) -> P V and S (1,030) and the hand-overs between them.  One query tile per CTA with two
// threads a row took 2,500 clocks for half the work, most of it instructions of the one producer (two 64-bit divisions
// and eight boxes a tile) and of the issuer (unrolled per case, fetched anew every tile): K and V have a producer each
// now, boxes are found 32 at a time, and the issuer is one short loop.  4096 tokens over 12000, 32 / 8 heads: 1,115 ->
// 736 us (1.28 PFLOP/s, power-capped); 8 x 1500: 318 -> 193; 3 x 3000 with remainders 440 -> 300, windowed 320 -> 205.
// Two issuers, one per query tile, were slower (975 us free-running, as both tiles then wait for the same unit; 839 in
// turns), and so were two threads a row (874 against 849).
// The reference maximum is only moved when a row's maximum grows by more than 2^8 (then that warp
// rescales its O rows in TMEM), so O is read from TMEM once, at the end.
// Where the query tiles leave SMs idle, a cluster of CTAs shares the K/V tiles of a pair of query tiles: each leaves its
// unnormalised O, reference maxima and row sums in its shared memory, and each combines the ranks' results for a part of
// the rows.
// Warp roles: 2 x 4 softmax warps, 2 TMA producers (K and V pages gathered through the block table, one 4 KiB
// box per 16-token page slab, 128-byte swizzle, no multicast), 1 MMA issuer that also owns
// the TMEM allocation.  Every wait is bounded and reports MIE_STATUS_WAIT_TIMEOUT.
#pragma once

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "umma.cuh"

namespace mie {
namespace {

constexpr int kRows = 128;                       // rows of a query tile (tokens x group heads)
constexpr int kTiles = 2;                        // query tiles per CTA
constexpr int kKv = 128;                         // K/V tokens per tile
constexpr int kSub = 16;                         // tokens per TMA box
constexpr int kBoxes = kKv / kSub;
constexpr int kTileWarps = 4;                    // softmax warps per query tile: one thread per row
constexpr int kSoftmaxWarps = kTiles * kTileWarps;
constexpr int kKWarp = kSoftmaxWarps, kVWarp = kSoftmaxWarps + 1, kMmaWarp = kSoftmaxWarps + 2;
constexpr int kThreads = (kSoftmaxWarps + 4) * 32;  // and an idle warp: whole warpgroups for setmaxnreg
// Registers a thread: a softmax thread holds a whole row of S.  384 threads start with 168 (64,512 in all); 2 x 128
// threads with 216 and 128 with 72 are as many.
constexpr int kSoftmaxRegs = 216, kOtherRegs = 72;
constexpr float kRescaleThreshold = 8.0f;        // log2 units
constexpr int kSmemLimit = 227 * 1024;
constexpr int kMaxSplit = 8;                     // CTAs that share a pair of query tiles
constexpr int kMinTiles = 4;                     // K/V tiles that are worth a rank of a split

// Shared memory (1024-byte aligned): Q tiles | K ring | V ring | barriers.
// A K tile has KH, a V tile VH groups of 64 dims.  Two layouts of a tile, both 128-byte swizzled with 8-token
// core groups of 1 KiB per 64 dims:
//   slab   [token / 8][dim / 64][token % 8][64 dims]  one 5-D box lands 16 whole tokens (head size a multiple of 64)
//   split  [dim / 64][token / 8][token % 8][64 dims]  one 4-D box per 64 dims, a partial last group zero-filled by TMA
template <int KH, int VH>
struct PrefillTile {
  static constexpr int kQTile = kRows * KH * 128;  // bytes
  static constexpr int kKTile = kKv * KH * 128;
  static constexpr int kVTile = kKv * VH * 128;
  static constexpr int kRoom = kSmemLimit - 2048 - kTiles * kQTile;  // for both rings
  // Up to three stages each; where they don't fit, two of V before a second of K: K(j+1) has the time of a softmax to
  // arrive once S(j) has read K(j), V(j+1) only that of S(j+1) once P(j) V(j) has read V(j).
  static constexpr int kKStages = kRoom >= 3 * kKTile + 2 * kVTile ? 3 : kRoom >= 2 * kKTile + 2 * kVTile ? 2 : 1;
  static constexpr int kVRoom = (kRoom - kKStages * kKTile) / kVTile;
  static constexpr int kVStages = kVRoom >= 3 ? 3 : kVRoom;
  static constexpr int kOffK = kTiles * kQTile;
  static constexpr int kOffV = kOffK + kKStages * kKTile;
  static constexpr int kOffBar = kOffV + kVStages * kVTile;
  // Of a split: O of both query tiles, VH * 64 floats a row, over everything before the barriers, and reference maximum
  // and sum of each row (in the last ring stage, behind O).
  static constexpr int kOffState = kTiles * kRows * VH * 256;
  static constexpr int kOffWeight = kOffState + kTiles * kRows * 16;  // [rank][row] floats
  static constexpr int kSmemBytes = kOffBar + 256 + 1024;
  static_assert(kVStages >= 1 && kSmemBytes <= kSmemLimit, "one CTA's shared memory");
  static_assert(kOffWeight + kMaxSplit * kTiles * kRows * 4 <= kOffBar, "the state of a split fits over Q and the rings");
};

struct UmmaPrefillParams {
  const char* query;
  long long q_st, q_sh;
  char* out;
  long long o_st, o_sh;
  IndexView tables, cu_seqlens, kv_lens;
  int requests, q_heads, kv_heads, group, block_size, num_blocks, table_width;
  float scale_log2;
  int* status;
  // The extended kernel only: head sizes, sliding window (0: none), sinks (null: none), passes over the value
  // dimensions (128 each), and which of K / V use the slab layout.
  int dim, vdim, v_passes, k_slab, v_slab;
  long long window;
  const float* sinks;
};

enum Bar { kQFull = 0, kKFull = 1, kKEmpty = 4, kVFull = 7, kVEmpty = 10, kSFull = 13, kPFull = 15, kODone = 19,
           kVClean = 21, kNumBars = 22 };

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
template <int kRegs>
__device__ __forceinline__ void raise_registers() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void lower_registers() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// 16 bytes from global to shared memory without waiting for them, or zeros.
__device__ __forceinline__ void copy16_or_zero(void* dst, const void* src, bool copy) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(copy ? 16 : 0)
               : "memory");
}

// 2^x on the special-function unit; -inf gives +0.
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// kExt = false: head_dim 128, plain softmax, probabilities rounded to the activation dtype.
// kExt = true: other head sizes (several passes over wide values), sliding window, sinks, and P V with the
// probabilities as a rounded part plus remainder, so that weights keep about 16 bits.
template <typename T, int KH, int VH, bool kExt>
__global__ void __launch_bounds__(kThreads, 1)
    prefill_umma_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                        const UmmaPrefillParams p, const int q_tiles, const int split) {
  using Tile = PrefillTile<KH, VH>;
  constexpr int kKStages = Tile::kKStages, kVStages = Tile::kVStages, kKTile = Tile::kKTile, kVTile = Tile::kVTile;
  constexpr int kOffK = Tile::kOffK, kOffV = Tile::kOffV, kOffBar = Tile::kOffBar;
  // Bytes between 8-token groups and between 64-dim groups of a K / V tile.
  const bool k_slab = !kExt || p.k_slab != 0, v_slab = !kExt || p.v_slab != 0;
  const uint32_t k_group = k_slab ? KH * 1024 : 1024, k_half = k_slab ? 1024 : kKv * 128;
  const uint32_t v_group = v_slab ? VH * 1024 : 1024, v_half = v_slab ? 1024 : kKv * 128;
  static_assert(!kExt || std::is_same<T, __nv_bfloat16>::value, "remainders are taken of bf16 probabilities");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;

  chain_release();
  chain_wait();
  const int r = blockIdx.y;
  const int kvh = kExt ? (int)blockIdx.z / p.v_passes : (int)blockIdx.z;
  const int v_box0 = kExt ? ((int)blockIdx.z % p.v_passes) * VH : 0;  // first 64-dim value group of this pass
  const int rank = (int)blockIdx.x % split;                // this CTA's part of the K/V tiles
  const int qt = q_tiles - 1 - (int)blockIdx.x / split;  // latest (heaviest) query tiles first
  const int tile_toks = kRows / p.group;
  const long long q_begin = p.cu_seqlens.at(r), q_end = p.cu_seqlens.at(r + 1);
  const int q_len = (int)(q_end - q_begin);
  const long long kv_len = p.kv_lens.at(r);
  int i0 = qt * kTiles * tile_toks;
  if (i0 >= q_len) return;
  if (kv_len < q_len || kv_len > (long long)p.table_width * p.block_size) {
    if (threadIdx.x == 0) raise_status(p.status, MIE_STATUS_BAD_LENGTH);
    return;
  }
  const long long offset = kv_len - q_len;  // position of query token 0
  // K/V tiles: the first that any row from token `tok` on sees (its own window starts latest back), and the one behind
  // the last that token `tok` sees.
  auto first_tile = [&](int tok) {
    return kExt && p.window > 0 && offset + tok + 1 > p.window ? (int)((offset + tok + 1 - p.window) / kKv) : 0;
  };
  auto end_tile = [&](int tok) { return (int)((offset + tok) / kKv) + 1; };
  // Live tokens of both query tiles; the second may be empty.
  const int left1 = q_len - i0 - tile_toks;
  int toks0 = left1 < 0 ? left1 + tile_toks : tile_toks, toks1 = left1 < 0 ? 0 : left1 < tile_toks ? left1 : tile_toks;
  int all0 = first_tile(i0), all = end_tile(i0 + (toks1 > 0 ? tile_toks + toks1 : toks0) - 1) - all0;
  // The ranks that share these tiles have at least kMinTiles each.  Too few to share: a rank per query tile.
  int ranks = all < split * kMinTiles ? (all < kMinTiles ? 1 : all / kMinTiles) : split;
  if (split > 1 && ranks == 1 && toks1 > 0) {
    if (rank > 1) return;
    if (rank == 1) i0 += tile_toks, toks0 = toks1;
    toks1 = 0;
    all0 = first_tile(i0), all = end_tile(i0 + toks0 - 1) - all0;
  } else if (rank >= ranks) {
    return;
  }
  const int part = ranks > 1 ? rank : 0;
  const int tile0 = all0 + (int)((long long)all * part / ranks);
  const int n_tiles = all0 + (int)((long long)all * (part + 1) / ranks) - tile0;
  // Each query tile's share of them; the first query tile's is never larger unless the second is empty.
  const int own0 = end_tile(i0 + toks0 - 1) - tile0;
  const int n0 = own0 < 0 ? 0 : own0 < n_tiles ? own0 : n_tiles, n1 = toks1 > 0 ? n_tiles : 0;

  if (threadIdx.x == 0) {
    mbar_init(&bars[kQFull], kSoftmaxWarps);
    for (int s = 0; s < kKStages; ++s) {
      mbar_init(&bars[kKFull + s], 1);
      mbar_init(&bars[kKEmpty + s], 1);
    }
    for (int s = 0; s < kVStages; ++s) {
      mbar_init(&bars[kVFull + s], 1);
      mbar_init(&bars[kVEmpty + s], 1);
    }
    for (int t = 0; t < kTiles; ++t) {
      mbar_init(&bars[kSFull + t], 1);
      mbar_init(&bars[kPFull + 2 * t], kTileWarps);
      mbar_init(&bars[kPFull + 2 * t + 1], kTileWarps);
      mbar_init(&bars[kODone + t], 1);
    }
    mbar_init(&bars[kVClean], 1);
    mbar_fence_init();
    tma_prefetch_desc(&kmap);
    tma_prefetch_desc(&vmap);
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Query tile t: S in columns [128 t, 128 t + 128), P written over the first 64 of them, its remainder (kExt) over
  // the other 64; O in columns 256 + 128 t and on.

  if (warp >= kSoftmaxWarps) {
  lower_registers<kOtherRegs>();
  if (warp == kKWarp || warp == kVWarp) {
    // ---------------- TMA producers: K tiles and V tiles (+ V tail sanitiser) ----------------
    const bool values = warp == kVWarp;
    const CUtensorMap* map = values ? &vmap : &kmap;
    const int stages = values ? kVStages : kKStages, tile_bytes = values ? kVTile : kKTile;
    const int groups = values ? VH : KH, box0 = values ? v_box0 : 0;
    const bool slab = values ? v_slab : k_slab;
    uint8_t* ring = smem + (values ? kOffV : kOffK);
    uint64_t* full = &bars[values ? kVFull : kKFull];
    uint64_t* empty = &bars[values ? kVEmpty : kKEmpty];
    const uint64_t policy = l2_evict_first_policy();
    // Where the boxes of four tiles are, one box of 16 tokens per lane, requested four tiles ahead: no load waits for a
    // lookup, and the divisions are done once per box.  Boxes past the request's length still land (page 0), so that a
    // stage always receives the same byte count; their scores are masked and their V rows zeroed below.
    struct Box {
      int page, row;  // tensor-map coordinates
    };
    const unsigned page_boxes = (unsigned)p.block_size / kSub;
    auto find_boxes = [&](int group) {
      Box at{0, slab ? kvh * (p.block_size / 8) : 0};
      const long long box = (long long)tile0 * kBoxes + group * 32 + lane;
      if (group * 4 + lane / kBoxes >= n_tiles || box * kSub >= kv_len) return at;
      const unsigned page = (unsigned)box / page_boxes, in_page = ((unsigned)box - page * page_boxes) * kSub;
      const long long id = p.tables.at(r, page);
      if (id < 0 || id >= p.num_blocks) {
        raise_status(p.status, MIE_STATUS_BAD_PAGE);
        return at;
      }
      at.page = (int)id;
      at.row += slab ? in_page / 8 : in_page;
      return at;
    };
    Box here = find_boxes(0), next = find_boxes(1);
    int s = 0;
    uint32_t parity = 1;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      if (j % 4 == 0 && j > 0) {
        here = next;
        next = find_boxes(j / 4 + 1);
      }
      const int from = j % 4 * kBoxes + lane % kBoxes;
      const int page = __shfl_sync(0xffffffffu, here.page, from), row = __shfl_sync(0xffffffffu, here.row, from);
      ok = warp_wait_bounded(&empty[s], parity);
      if (!ok) break;
      if (elect_one()) mbar_expect_tx(&full[s], tile_bytes);
      __syncwarp();
      if (lane < kBoxes) {
        uint8_t* dst = ring + s * tile_bytes;
        if (slab) {
          tma_load_5d_hint(dst + lane * (tile_bytes / kBoxes), map, &full[s], 0, 0, box0, row, page, policy);
        } else {
          for (int x = 0; x < groups; ++x)
            tma_load_4d_hint(dst + x * (kKv * 128) + lane * (kSub * 128), map, &full[s], (box0 + x) * 64, row, kvh, page,
                             policy);
        }
      }
      __syncwarp();
      if (++s == stages) s = 0, parity ^= 1u;
    }
    if (ok && values) {
      // Slots past the request's length may hold anything (even NaN bits): zero those V rows of the last
      // tile so that a zero probability times V stays zero, then tell the MMA warp the stage is clean.
      const int last = n_tiles - 1, stage = last % kVStages;
      ok = warp_wait_bounded(&full[stage], (last / kVStages) & 1u);
      if (ok) {
        const long long first_bad = kv_len - ((long long)tile0 + last) * kKv;  // rows >= first_bad are past the length
        uint8_t* vdst = ring + stage * kVTile;
        for (int c = lane; c < kKv * VH * 8; c += 32) {
          const int row = c / (VH * 8), chunk = c % (VH * 8);
          if (row >= first_bad)
            *reinterpret_cast<uint4*>(vdst + (row >> 3) * v_group + (chunk >> 3) * v_half + (row & 7) * 128 +
                                      (chunk & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[kVClean]);
      }
    }
    if (!ok && lane == 0) raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer ----------------
    // One copy of the code for both query tiles, descriptors by one addition each: this warp's instructions, fetched
    // anew between those of the softmax warps, are on the path between P and the next S.
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t idesc_s = instr_desc_f16(kKv, kFmt, 0);      // S = Q K^T: both K-major in shared memory
    constexpr uint32_t idesc_o = instr_desc_f16(VH * 64, kFmt, 1);  // O += P V : A = P in TMEM, B = V, MN-major
    const uint64_t q_desc0 = smem_desc_k128(smem_u32(smem));
    const uint64_t k_desc0 = smem_desc_k128(smem_u32(smem + kOffK), k_group);
    const uint64_t v_desc0 = smem_desc_mn128(smem_u32(smem + kOffV), v_half, v_group);
    // S(t, j) overwrites the columns of P(t, j-1): P(t, j-1) V(j-1) was issued before by this thread and tcgen05.mma
    // executes in issue order, so no barrier is needed.  For the same reason S(t, j) complete means that O holds
    // every tile before j.
    auto issue_s = [&](int t, int s, bool last) {
      tc_fence_after();
      if (elect_one()) {
        const uint64_t q_desc = q_desc0 + t * (Tile::kQTile >> 4), k_desc = k_desc0 + s * (kKTile >> 4);
        const uint32_t tmem_s = tmem_base + t * kKv;
#pragma unroll
        for (int ks = 0; ks < KH * 4; ++ks) {  // 16 dims each
          if (kExt && ks * 16 >= p.dim) break;
          umma_f16(tmem_s, q_desc + (((ks >> 2) * (kRows * 128) + (ks & 3) * 32) >> 4),
                   k_desc + (((ks >> 2) * k_half + (ks & 3) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
        }
        umma_commit(&bars[kSFull + t]);
        if (last) umma_commit(&bars[kKEmpty + s]);  // K stage free once these MMAs have read it
      }
      __syncwarp();
    };
    // Query tile 1 is the last to use a K/V tile unless it is empty.
    bool ok = warp_wait_bounded(&bars[kQFull], 0) && warp_wait_bounded(&bars[kKFull], 0);
    if (ok) {
#pragma unroll 1
      for (int t = n0 > 0 ? 0 : 1; t < (n1 > 0 ? 2 : 1); ++t) issue_s(t, 0, t == 1 || n1 == 0);
    }
    int ks = 0, vs = 0;  // stages of K(j) and V(j)
    uint32_t k_parity = 0, v_parity = 0;
#pragma unroll 1
    for (int j = 0; j < n_tiles && ok; ++j) {
      // What was loaded is waited for before P, whose arrival is what the products wait for.
      const int vs_now = vs;
      if (++ks == kKStages) ks = 0, k_parity ^= 1u;
      ok = warp_wait_bounded(&bars[kVFull + vs], v_parity) &&
           (j + 1 < n_tiles ? kKStages == 1 || warp_wait_bounded(&bars[kKFull + ks], k_parity)
                            : warp_wait_bounded(&bars[kVClean], 0));
      if (++vs == kVStages) vs = 0, v_parity ^= 1u;
#pragma unroll 1
      for (int t = 0; t < 2 && ok; ++t) {
        const int n_own = t == 0 ? n0 : n1;
        const bool last = t == 1 || n1 == 0;
        if (j >= n_own) continue;
        const uint32_t tmem_p = tmem_base + t * kKv, tmem_o = tmem_base + 256 + t * 128;
        // P comes in halves of 64 keys, so that the product starts while the second half's exponentials are computed.
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ok = warp_wait_bounded(&bars[kPFull + 2 * t + h], j & 1u);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t v_desc = v_desc0 + vs_now * (kVTile >> 4);
#pragma unroll
            for (int kt = h * kBoxes / 2; kt < (h + 1) * kBoxes / 2; ++kt) {  // 16 tokens = 8 TMEM columns of packed P
              const uint64_t db = v_desc + kt * (v_group >> 3);
              umma_f16_ts(tmem_o, tmem_p + kt * 8, db, idesc_o, (j > 0 || kt > 0) ? 1u : 0u);
              if (kExt) umma_f16_ts(tmem_o, tmem_p + 64 + kt * 8, db, idesc_o, 1u);  // the remainders
            }
            if (h == 1 && last) umma_commit(&bars[kVEmpty + vs_now]);  // V stage free once these MMAs have read it
            if (h == 1 && j == n_own - 1) umma_commit(&bars[kODone + t]);
          }
          __syncwarp();
        }
        if (ok && j + 1 < n_own) {
          // One stage: K(j + 1) could not be waited for above, where S(1, j) had yet to read K(j).  The first query tile to
          // use it waits, which is the second one when the first has had its last K/V tile.
          if (kKStages == 1 && (t == 0 || j + 1 >= n0)) ok = warp_wait_bounded(&bars[kKFull], k_parity);
          if (ok) issue_s(t, ks, last);
        }
      }
    }
    if (!ok && lane == 0) raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
  }
  } else {
    raise_registers<kSoftmaxRegs>();
    // ---------------- Softmax warps: one thread per query row ----------------
    const int t = warp / kTileWarps, quad = warp % kTileWarps;
    const int row = quad * 32 + lane;  // TMEM lane = row of the tile
    const int toks = t == 0 ? toks0 : toks1, n_own = t == 0 ? n0 : n1;
    const int first_tok = i0 + t * tile_toks;
    const int tok_local = row / p.group, head_local = row % p.group;
    const bool row_live = tok_local < toks;
    const long long first_pos = offset + first_tok;  // smallest query position of the tile
    const long long last_key = first_pos + toks - 1;
    const long long pos = row_live ? first_pos + tok_local : last_key;  // dead rows compute harmlessly
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t tmem_s = tmem_base + t * kKv + lane_addr, tmem_o = tmem_base + 256 + t * 128 + lane_addr;
    const long long own_q = (q_begin + first_tok + (row_live ? tok_local : 0)) * p.q_st +
                            (long long)(kvh * p.group + (row_live ? head_local : 0)) * p.q_sh;
    const uint32_t live_rows = __ballot_sync(0xffffffffu, row_live);
    if (n_own > 0) {
      // This warp's 32 query rows into shared memory, KH * 8 lanes a row, K-major with the 128-byte swizzle of a K tile;
      // rows past the chunk and dims past the head size are zero.
      uint8_t* tile = smem + t * Tile::kQTile + quad * 32 * 128;
#pragma unroll 4
      for (int i = lane; i < 32 * KH * 8; i += 32) {
        const int x = i / (KH * 8), c = i % (KH * 8);
        const long long at = __shfl_sync(0xffffffffu, own_q, x);
        const bool in = (live_rows >> x & 1) && (!kExt || c * 8 < p.dim);
        copy16_or_zero(tile + (c >> 3) * (kRows * 128) + x * 128 + (((c ^ x) & 7) << 4),
                       reinterpret_cast<const T*>(p.query) + (in ? at + c * 8 : 0), in);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      fence_proxy_async_smem();
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[kQFull]);
    // m_ref lives in the scaled log2 domain (score * scale * log2 e); scale > 0 is checked on the host, so
    // the row maximum can be taken over the raw scores.
    const float scale = p.scale_log2;
    float m_ref = -INFINITY, l = 0.f;
    const bool sunk = kExt && p.sinks != nullptr && part == 0;
    if (sunk) {
      // The sink opens the softmax: reference maximum and one unit of denominator.
      m_ref = row_live ? p.sinks[kvh * p.group + head_local] * 1.4426950408889634f : 0.f;
      l = 1.f;
    }
    // Tiles from `masked_from` on have keys that some row may not see at their end, those before `windowed_to` at their
    // start.
    const long long base = (long long)tile0 * kKv;
    const int masked_from = (int)((first_pos - base + 1) / kKv);
    const int windowed_to =
        kExt && p.window > 0 && last_key >= p.window + base ? (int)((last_key - p.window - base) / kKv) + 1 : 0;
    bool ok = true;
    for (int j = 0; j < n_own; ++j) {
      if (!mbar_wait_bounded(&bars[kSFull + t], j & 1u)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      float sv[kKv];
#pragma unroll
      for (int c = 0; c < kKv; c += 32) tmem_ld32(tmem_s + c, *reinterpret_cast<float(*)[32]>(&sv[c]));
      tmem_ld_wait();
      if (j >= masked_from) {
        // Only tiles that reach the causal diagonal (or the end of the request) carry masked keys.
        const long long d = pos - base - (long long)j * kKv;
        const int lim = d < -1 ? -1 : d < kKv ? (int)d : kKv;  // keys [0, lim] are visible
        const int all_see = __reduce_min_sync(0xffffffffu, lim);
#pragma unroll
        for (int c = 0; c < kKv; c += 32) {
          if (all_see >= c + 31) continue;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i > lim) sv[c + i] = -INFINITY;
        }
      }
      if (kExt && j < windowed_to) {
        // Tiles that reach back past some row's window: keys before `lo` are hidden.
        const long long d = pos - p.window + 1 - base - (long long)j * kKv;
        const int lo = d < 0 ? 0 : d > kKv ? kKv : (int)d;
        const int some_hide = __reduce_max_sync(0xffffffffu, lo);
#pragma unroll
        for (int c = 0; c < kKv; c += 32) {
          if (some_hide <= c) break;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c + i < lo) sv[c + i] = -INFINITY;
        }
      }
      float mx4[4] = {sv[0], sv[1], sv[2], sv[3]};
#pragma unroll
      for (int c = 4; c < kKv - 4; c += 8) {
#pragma unroll
        for (int q = 0; q < 4; ++q) mx4[q] = max3(mx4[q], sv[c + 2 * q], sv[c + 2 * q + 1]);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) mx4[q] = max3(mx4[q], sv[kKv - 4 + 2 * q], sv[kKv - 3 + 2 * q]);
      const float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * scale;
      // Move the reference maximum only on the first tile or when a row outgrew it by 2^8.
      const bool grow = mx > m_ref + kRescaleThreshold || (j == 0 && !sunk);
      if (__any_sync(0xffffffffu, grow)) {
        float alpha = 1.f;
        if (grow) {
          const float m_new = fmaxf(m_ref, mx);
          // 0 on the first tile; a row may have seen no key yet (both maxima -inf) with a window or a split.
          alpha = m_new == -INFINITY ? 1.f : ex2_approx(m_ref - m_new);
          m_ref = m_new;
        }
        l *= alpha;
        if (j > 0) {
          // Rescale this warp's 32 rows of O in TMEM (rows that did not grow use alpha = 1).  O holds every tile before
          // this one: S(j) was issued behind them.
#pragma unroll 1
          for (int c = 0; c < VH * 64; c += 16) {
            float ov[16];
            tmem_ld16(tmem_o + c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) ov[i] *= alpha;
            tmem_st16(tmem_o + c, *reinterpret_cast<const uint32_t(*)[16]>(&ov));
          }
        }
      }
      const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
      const float2 scale2 = make_float2(scale, scale), neg_m2 = make_float2(-m_use, -m_use);
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < kKv; c += 32) {  // 32 keys = 16 packed columns
        uint32_t w[16], rest[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          float2 e = __ffma2_rn(make_float2(sv[c + 2 * q], sv[c + 2 * q + 1]), scale2, neg_m2);
          e.x = ex2_approx(e.x);
          e.y = ex2_approx(e.y);
          sum2[q & 1] = __fadd2_rn(sum2[q & 1], e);
          w[q] = Mma16816<T>::pack(e.x, e.y);
          if (kExt) {  // what the rounding took away (bf16: the upper halves of two floats)
            const float2 kept = make_float2(__uint_as_float(w[q] << 16), __uint_as_float(w[q] & 0xffff0000u));
            const float2 lost = __ffma2_rn(kept, make_float2(-1.f, -1.f), e);
            rest[q] = Mma16816<T>::pack(lost.x, lost.y);
          }
        }
        tmem_st16(tmem_s + c / 2, w);
        if (kExt) tmem_st16(tmem_s + 64 + c / 2, rest);
        if (c % 64 == 32) {
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[kPFull + 2 * t + c / 64]);
        }
      }
      l += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
    }
    if (ok && n_own > 0) ok = mbar_wait_bounded(&bars[kODone + t], 0);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) raise_status(p.status, MIE_STATUS_WAIT_TIMEOUT);
    tc_fence_after();
    const int d0 = v_box0 * 64;  // first output dim of this pass
    if (ranks == 1) {
      // Rows through shared memory, so that the lanes of a row write it together: over this query tile's own Q, which is
      // done with, in passes where it is narrower than the output (the other tile may still have products to come).
      const float inv = 1.f / fmaxf(l, 1.17549435e-38f);
      const long long own_o = (q_begin + first_tok + (row_live ? tok_local : 0)) * p.o_st +
                              (long long)(kvh * p.group + (row_live ? head_local : 0)) * p.o_sh;
      constexpr int kGroups = KH < VH ? KH : VH, kChunks = kGroups * 8;  // of a pass: 64-dim groups, 16-byte chunks a row
      static_assert(VH % kGroups == 0 && kRows * kChunks * 16 <= Tile::kQTile, "a pass fits the tile's own Q");
      if (ok && n_own > 0) {
        uint8_t* rows = smem + t * Tile::kQTile + quad * (32 * kChunks * 16);
#pragma unroll 1
        for (int first = 0; first < VH * 64; first += kGroups * 64) {
          if (first > 0) __syncwarp();  // the last pass's rows have been read
#pragma unroll 1
          for (int c = 0; c < kGroups * 64; c += 32) {
            float ov[32];
            tmem_ld32(tmem_o + first + c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint32_t w[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) w[q] = Mma16816<T>::pack(ov[i + 2 * q] * inv, ov[i + 2 * q + 1] * inv);
              *reinterpret_cast<uint4*>(rows + (lane * kChunks + (((c + i) / 8 ^ lane) & (kChunks - 1))) * 16) =
                  make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
          __syncwarp();
          const int d = d0 + first;
#pragma unroll 4
          for (int i = lane; i < 32 * kChunks; i += 32) {
            const int x = i / kChunks, c = i % kChunks;
            const long long at = __shfl_sync(0xffffffffu, own_o, x);
            if ((live_rows >> x & 1) && (!kExt || d + c * 8 < p.vdim))
              *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + at + d + c * 8) =
                  *reinterpret_cast<const uint4*>(rows + (x * kChunks + ((c ^ x) & (kChunks - 1))) * 16);
          }
        }
      }
    } else {
      // This rank's part of the softmax: O rows over Q and the rings (both query tiles' products are done with them),
      // 16-byte chunks swizzled by the row; reference maximum and sum behind them.  A rank that had no K/V tile for a query
      // tile, or whose wait failed, counts for nothing.
      constexpr int kChunks = VH * 16, kORow = VH * 256;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      uint8_t* mine = smem + t * (kRows * kORow);
      const bool counts = ok && n_own > 0;
#pragma unroll 1
      for (int c = 0; c < VH * 64; c += 32) {
        if (!counts) break;
        float ov[32];
        tmem_ld32(tmem_o + c, ov);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4*>(mine + row * kORow + (((c / 4 + i) ^ row) & (kChunks - 1)) * 16) =
              make_float4(ov[4 * i], ov[4 * i + 1], ov[4 * i + 2], ov[4 * i + 3]);
      }
      *reinterpret_cast<float4*>(smem + Tile::kOffState + (t * kRows + row) * 16) =
          make_float4(counts ? m_ref : -INFINITY, counts ? l : 0.f, counts ? 1.f : 0.f, 0.f);
      __syncwarp();
      cluster_sync_all();
      const uint32_t local = smem_u32(smem);
      float* weights = reinterpret_cast<float*>(smem + Tile::kOffWeight);
      {  // what each rank's row counts for in the result, a thread a row; -1: it has no such row
        float top = -INFINITY, sum = 0.f;
        float4 v[kMaxSplit];  // reference maximum, sum, whether it counts
#pragma unroll
        for (int i = 0; i < kMaxSplit; ++i) {
          v[i] = i < ranks ? ld_cluster_f4(local + Tile::kOffState + threadIdx.x * 16, i)
                           : make_float4(-INFINITY, 0.f, 0.f, 0.f);
          top = fmaxf(top, v[i].x);
        }
        // A rank whose keys are all hidden from the row, or all NaN, has -inf as its maximum: the weight is 0, and what is
        // not a number in its sum (or, below, in its values) still reaches the result, as it does without a split.
#pragma unroll
        for (int i = 0; i < kMaxSplit; ++i) {
          v[i].x = v[i].x == -INFINITY ? 0.f : ex2_approx(v[i].x - top);
          sum += v[i].y * v[i].x;
        }
        const float inv = sum != sum ? sum : 1.f / fmaxf(sum, 1.17549435e-38f);
#pragma unroll
        for (int i = 0; i < kMaxSplit; ++i)
          weights[i * (kTiles * kRows) + threadIdx.x] = v[i].z != 0.f ? v[i].x * inv : -1.f;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // VH * 16 lanes combine a row, 4 dims a lane; the ranks share the live rows.  A remote load takes about 1,300 clocks,
      // so sixteen are in flight: of all ranks, and of several rows.
      constexpr int kLanes = kChunks, kStep = kSoftmaxWarps * 32 / kLanes;
      const int chunk = threadIdx.x % kLanes, d = v_box0 * 64 + chunk * 4;
      const int live0 = toks0 * p.group, live = live0 + toks1 * p.group;
      auto combine = [&](auto rank_count, auto row_count) {
        constexpr int kRanks = rank_count.value, kBatch = row_count.value;
        for (int y0 = rank + ranks * ((int)threadIdx.x / kLanes); y0 < live; y0 += ranks * kStep * kBatch) {
          int x[kBatch];
          float4 v[kBatch][kRanks];
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            const int y = y0 + b * ranks * kStep < live ? y0 + b * ranks * kStep : y0;
            x[b] = y < live0 ? y : kRows + y - live0;
#pragma unroll
            for (int i = 0; i < kRanks; ++i)
              v[b][i] = ld_cluster_f4(local + x[b] * kORow + ((chunk ^ x[b]) & (kLanes - 1)) * 16, i < ranks ? i : rank);
          }
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kRanks; ++i) {
              const float w = weights[i * (kTiles * kRows) + x[b]];
              if (!(w < 0.f))
                o.x += v[b][i].x * w, o.y += v[b][i].y * w, o.z += v[b][i].z * w, o.w += v[b][i].w * w;
            }
            if (y0 + b * ranks * kStep >= live || (kExt && d >= p.vdim)) continue;
            const int t = x[b] / kRows, tok = x[b] % kRows / p.group, head = x[b] % kRows % p.group;
            T* out = reinterpret_cast<T*>(p.out) + (q_begin + i0 + t * tile_toks + tok) * p.o_st +
                     (long long)(kvh * p.group + head) * p.o_sh + d;
            *reinterpret_cast<uint2*>(out) =
                make_uint2(Mma16816<T>::pack(o.x, o.y), Mma16816<T>::pack(o.z, o.w));
          }
        }
      };
      if (ranks == 2)
        combine(std::integral_constant<int, 2>(), std::integral_constant<int, 8>());
      else if (ranks <= 4)
        combine(std::integral_constant<int, 4>(), std::integral_constant<int, 4>());
      else
        combine(std::integral_constant<int, 8>(), std::integral_constant<int, 2>());
    }
  }

  if (ranks > 1) {
    __syncwarp();
    if (warp >= kSoftmaxWarps) cluster_sync_all();
    cluster_sync_all();  // nobody's shared memory goes before all have read it
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// CTAs that share the K/V tiles of a pair of query tiles: as many as leave all clusters on the GPU at once (of 148 SMs 74
// clusters of two, 33 of four, 15 of eight; the 16 heads of a short prompt as clusters of eight take a second round: 64 tokens
// with 192-dim keys 10.4 us, as clusters of four 9.5; one token over 4100 31.6 and 20.7).  16 tokens over 3000: 38 us unsplit,
// 14 with six CTAs; 386 and 126 tokens over 1024: 31 us and 24; what it costs is 3 to 5 us (the ranks' O through remote shared
// memory), which eight tiles in two halves pay.  75 to 148 pairs are only split where the wait of the last is no loss (below);
// else a pair of the longest rows takes longer than two CTAs with a query tile each did.  Clusters of two of which only the
// heaviest pairs use both are no way out: the SM that an idle rank leaves is not given to another cluster (20 -> 40 us).
template <typename T, int KH, int VH, bool kExt>
int launch_prefill(const CUtensorMap& kmap, const CUtensorMap& vmap, const UmmaPrefillParams& p, long long tokens,
                   int max_query_len, cudaStream_t stream) {
  constexpr int kSmem = PrefillTile<KH, VH>::kSmemBytes;
  const auto kernel = prefill_umma_kernel<T, KH, VH, kExt>;
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kSmem;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  const auto in_clusters = [&](int size) {
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = (unsigned)size;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    return a;
  };
  static std::atomic<bool> configured[64];
  static int fitting[64][4];  // clusters of 2, 4 and 8 that the device holds
  int dev = 0;
  MIE_CUDA(cudaGetDevice(&dev));
  MIE_CHECK_ARG(dev >= 0 && dev < 64, "device %d", dev);
  if (!configured[dev].load(std::memory_order_acquire)) {
    MIE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    config.attrs = attr;
    config.numAttrs = 1;
    for (int i = 1; i < 4; ++i) {
      attr[0] = in_clusters(1 << i);
      config.gridDim = dim3(1u << i);
      MIE_CUDA(cudaOccupancyMaxActiveClusters(&fitting[dev][i], kernel, &config));
    }
    configured[dev].store(true, std::memory_order_release);
  }
  const int pair_tokens = kTiles * (kRows / p.group);
  const int q_tiles = (max_query_len + pair_tokens - 1) / pair_tokens;
  const int columns = p.kv_heads * (kExt ? p.v_passes : 1);
  // Pairs with live rows, as far as the host knows: as many as there can be when the requests are about equally long.  Of
  // ragged ones the last pair is half empty on average, and each has one; that counts short requests for less than a pair,
  // but theirs are over soon.
  const long long most = (long long)q_tiles * p.requests, mean = tokens / pair_tokens + (p.requests + 1) / 2;
  const bool equal = tokens * 16 >= (long long)max_query_len * p.requests * 15;
  const long long likely = (equal || mean > most ? most : mean < p.requests ? p.requests : mean) * columns;
  int split = 1;
  for (int i = 1; i < 4 && likely <= fitting[dev][i]; ++i) split = 1 << i;
  // Prompts with little room for a prefix: a pair has half of the last one's K/V tiles on average, and clusters of two that
  // have to wait are over before the longest if they are the lighter pairs of the last (request, head), which come last, or of
  // the last two of eight and more for a whole prompt of many tiles.  3000 tokens of 8 heads on one (94 pairs) 45.1 -> 32.0 us, of 8 heads on 8
  // (96) 44.8 -> 41.5; left alone: two of 1500 on 8 (96) 27.2 -> 32.5, three of 3000 of 4 on one (141) 45.7 -> 51.2.
  const long long room = (long long)p.table_width * p.block_size, waiting = likely - fitting[dev][1];
  const int tiles = max_query_len / kKv;
  const bool two = 8 * room <= 9ll * max_query_len && tiles >= 16 && 4 * q_tiles <= fitting[dev][1];
  if (split == 1 && likely <= sm_count() && equal && tiles >= 12 && waiting <= (two ? 2 : 1) * q_tiles &&
      2 * room <= 3ll * max_query_len && (p.window == 0 || p.window >= max_query_len))
    split = 2;
  config.gridDim = dim3((unsigned)(q_tiles * split), (unsigned)p.requests, (unsigned)columns);
  config.attrs = attr;
  config.numAttrs = 0;
  if (chained_launch_enabled()) {
    attr[config.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[config.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (split > 1) attr[config.numAttrs++] = in_clusters(split);
  MIE_CUDA(cudaLaunchKernelEx(&config, kernel, kmap, vmap, p, q_tiles, split));
  MIE_LAUNCH_CHECK("prefill_umma_kernel");
  return MIE_OK;
}

}  // namespace

// Defined in prefill_attention_umma.cu: cached 5-D slab map over pages [page, head, token, dim] (dim a multiple of
// 64) whose box is 16 tokens x `box_groups` 64-dim groups, and whether a page layout allows it.
int page_slab_map(const mie_view4_t& pages, int num_blocks, int kv_heads, int block_size, int dim, int box_groups,
                  int dtype, CUtensorMap* out);
bool pages_fit_slab_map(const mie_view4_t& v, int block_size, int dim);

}  // namespace mie
