// FP8 block-scaled GEMM for sm_100a: TMA-fed shared-memory ring, tcgen05.mma
// (kind::f8f6f4) into double-buffered TMEM partials, and an fp32 promotion of
// every 128-deep K-block partial by a_scale * b_scale in the epilogue warps.
//
// Computes what ks_gemm_fp8_blockwise / _nt / ks_moe_grouped_gemm_fp8_blockwise
// declare, for block_n = block_k = 128 (reference algebra:
// kernels/src/gemm/gemm_fp8_blockwise.cu:107-150 — an fp32 inner product per
// K-block, folded into the fp32 output with the block's scale product).
//
// CTA anatomy (one CTA per SM, persistent over output tiles of 128 x BN):
//   warp 0      TMA producer: A tile 128 x 128 B and B tile BN x 128 B per stage,
//               128-byte swizzle, completion counted on the stage's `full` barrier
//   warp 1      MMA issuer: 4 UMMAs (M128, N=BN, K32) per K-block into one of the TMEM
//               accumulator buffers (two of 256 columns, four of 128); ONE
//               tcgen05.commit per K-block both releases the stage to the producer
//               and tells the epilogue that the partial product is complete
//   warps 2,3   schedule: walk the tiles ahead of the epilogue and hand it every K-block's
//               a_scale * b_scale products and every tile's place through shared memory
//   warps 4-11  epilogue: warp w reads TMEM lanes 32*(w%4).. and BN/2 columns in
//               16-column loads, double-buffered so that one load is in flight
//               while the previous one is folded in:
//               acc = fma(partial, a_scale[row,kb] * b_scale[kb,nb], acc) in
//               registers (packed two-wide), frees the TMEM buffer, and after
//               the last K-block rounds once to the output type; the tile is turned
//               round in shared memory and stored in whole row segments.
// Last partial round of a dense problem: when T tiles leave T mod #CTAs tiles for a final
// round that would keep most SMs idle (896 tiles on 148 SMs: 8 tiles, 140 idle SMs for a
// whole tile time), those tiles are cut along K into S parts (S <= 8, parts x tiles <=
// #CTAs), each a CTA's first work item. A part's epilogue warps write their fp32 partial to
// a slot; split_reduce_kernel, launched behind the GEMM on the same stream, adds the parts in
// part order (reproducible) and writes the tiles. (Letting the last part to arrive reduce a
// tile inside the GEMM kernel measured 3-4 % gain instead of the 10 % the idle round costs:
// one CTA then reads S x 128 KB behind a fence and four dependent atomics while its tensor
// core waits.) Grouped problems, whose rounds only the device knows, are not cut: a row's sum would then depend on
// the other rows of the call, and the call would need slots and counters, in a captured graph too (8 experts, K=14336,
// N=4096, 16 bits: 205 us, 180 when cut).
// What bounds it: the epilogue warps' chain per K-block (wait, TMEM loads, 64 two-wide FMAs, release) and, back to
// back, the card's power limit. Per K-block of 128 x 256 x 128 the MMAs need 512 cycles; the loop took 872 while the
// epilogue warps loaded scales from global memory (a load over 32 lines per warp), looked for their next tile
// and stored by TMA piece by piece, 727 since warps 2 and 3 do the first two (M=4096, N=K=7168; with 28
// K-blocks a tile and f32 results 994 -> 881, 4096 tokens over 256 experts, N=7168, K=2048, 1340 -> 985).
// In time: M=4096, N=K=7168 alone 169 us (193 before), back to back 186 (200); SM clock 1.6 -> 1.5 GHz, the
// rest is power. The register budget decides: nothing of the K loop may be spilled (with one spilled value and 16-column
// loads 197 us, with two 200, with copies of the accumulators 240), so every address comes
// from one base, the tile's place is read again behind the loop, and no other wait stands in it.
// Measured and not better: 32-column loads (187), accumulators as 64-bit integers (240), handing the accumulator over
// in two 128-column halves (eight N=128 MMAs per K-block read A twice: 232), sixteen narrower epilogue
// warps, 224-wide tiles, scalar FMAs, paced MMA issue, sleeping or spinning waits.
// Problems with fewer tiles than SMs (decode: M = 16, N = 7168 is 28 tiles of 256 columns) are
// cut along K as well, over the S <= 8 CTAs of a cluster: each leaves its fp32 partial tile in
// its own shared memory (the ring is idle by then), and after a cluster barrier every CTA
// adds the S partials of its share of the tile's rows in part order, over distributed shared
// memory, and writes them. No scratch memory, no second kernel. S and the tile width are
// chosen in launch_fp8_blockwise(). Measured (cold L2): M=16, N=K=7168 28.7 -> 22.6 us; M=228,
// N=944, K=10256 38.9 -> 18.5; M=6, N=624, K=3712 16.4 -> 12.3; M=128, N=2048, K=7168 24.6 -> 16.4.
// B may be stored [N,K] (K-major UMMA operand) or [K,N] (MN-major operand, the
// layout of the reference C ABI); both are loaded by TMA without a transpose.
//
// Roofline: tensor-bound for M >= ~1024 (2*M*N*K flop over 4.5 PFLOP/s dense
// FP8); bytes per launch M*K + N*K + M*N*sizeof(out) + scales.
#include <mutex>
#include <optional>
#include <type_traits>

#include "common.cuh"
#include "sm100_fp8_gemm.cuh"
#include "sm100_fp8_store.cuh"
#include "sm100_host.cuh"
#include "sm100_ptx.cuh"

namespace ksb {
namespace sm100 {
namespace {

#ifndef KSB_FP8_ACC_BUFS_128
#define KSB_FP8_ACC_BUFS_128 4
#endif
#ifndef KSB_FP8_PANEL
#define KSB_FP8_PANEL 4
#endif

constexpr int kBM = 128;
constexpr int kBK = 128;
constexpr int kMaxExperts = 1024;
constexpr int kMaxOutParts = 8;

template <int BN>
struct Cfg {
  static constexpr int kStages = (BN == 256) ? 4 : 6;
  static constexpr int kABytes = kBM * kBK;
  static constexpr int kBBytes = BN * kBK;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // An epilogue warp owns 32 TMEM lanes x one of two column slices (a slot of the schedule holds the scales of two).
  static constexpr int kEpiCols = BN / 2;
  static constexpr int kEpiWarps = 8;
  static constexpr int kThreads = 128 + kEpiWarps * 32;
  // Warpgroup 0 (TMA, MMA issue) hands registers to the epilogue warpgroups,
  // which hold the accumulators plus the TMEM values in flight. The budgets must add up to no more than
  // the CTA's launch-time pool (threads x launch registers): setmaxnreg.inc
  // blocks, without a time limit, until the pool can satisfy it.
  static constexpr bool kRebalanceRegs = (BN == 256);
  // 12 warps, 168 registers at launch -> 40 / 232.
  static constexpr int kRegsIssue = 40;
  static constexpr int kRegsEpi = 232;
  // Accumulator buffers in TMEM (512 columns): the MMA warp runs this many K-blocks
  // ahead of the epilogue. A K-block's round trip (issue -> complete -> drained ->
  // handed back) is about 1400 cycles whatever the tile width, so narrow tiles,
  // whose MMAs are short, need more buffers in flight to keep the tensor core fed.
  static constexpr int kAccBufs = BN == 256 ? 2 : KSB_FP8_ACC_BUFS_128;
  static constexpr int kTmemCols = 512;
  // The finished tile is turned round in shared memory, 32 rows x 64 B per epilogue warp at a time.
  static constexpr int kPieceBytes = 64;
  static constexpr int kStagingBytes = kEpiWarps * 32 * kPieceBytes;
  static constexpr int kCtrlBytes = 512;   // barriers and flags
  // Slots of the schedule (see warps 2 and 3): a_scale * b_scale for the K-block's 128 rows and two column
  // slices. The tiles lie beside them: the schedule is at most kSlots tiles ahead of the one being stored.
  static constexpr int kSlots = 4;
  static constexpr int kSlotBytes = 2 * kBM * 4;
  static constexpr int kTileSlots = 8;
  static constexpr int kTileBytes = 32;
  static constexpr int kSchedBytes = kSlots * kSlotBytes + kTileSlots * kTileBytes;
  // ring + 1024 B alignment slack + store staging + barriers + slots, then the tile prefix, first rows
  // and end rows of the experts (grouped)
  static constexpr int smem_bytes(bool grouped) {
    return kStages * kStageBytes + 1024 + kStagingBytes + kCtrlBytes + kSchedBytes +
           (grouped ? 3 * 4 * (kMaxExperts + 1) : 0);
  }
};

struct Params {
  void* out;
  const float* a_scale;
  const float* b_scale;
  const int32_t* offsets;  // [E+1] when grouped
  unsigned int* fault_word;
  int num_experts;
  int m;        // rows of A (all experts together when grouped)
  int n, k;
  int nkb, nnb;
  int tiles_n;
  int tiles_m;  // dense only
  uint32_t idesc;
  int vec_store;  // 16-byte output stores are legal
  // K-split of the last partial round (dense only): work items [0, split_from) are whole
  // tiles; item split_from + r is part r % split_s of tile split_from + r / split_s.
  int split_from;
  int split_items;        // number of K-part items (tail tiles x split_s), at most the grid size
  int split_s;            // 1 = no split
  float4* split_slots;    // [tail tile][part][epilogue warp][16-byte column chunk][lane]
  int cluster_s;          // > 1: every tile is split (split_from = 0) over the CTAs of a cluster
  // MODE 1 / 2 (one scale per row and per column, the whole K range accumulated in TMEM)
  int64_t as_row_stride, as_kb_stride;   // a_scale[row * as_row_stride + kb * as_kb_stride]
  const void* bias;       // [N] in the output type or NULL
  int a_per_row;          // a_scale is [M] (else one value)
  int b_per_col;          // b_scale is [N] (else one value)
  // grouped, masked layout: expert e owns rows [e * max_m, e * max_m + masked_m[e])
  const int32_t* masked_m;
  int max_m;
  // scattered output (dense, 16-byte stores only): rows [b * rows_per_part, (b + 1) *
  // rows_per_part) are rows 0.. of out_parts[b]; 0 = one output
  int rows_per_part;
  void* out_parts[kMaxOutParts];
};

struct TileCoord {
  int expert, row0, row_end, n0;
  int kb0, kb1;   // K-blocks of this work item
  int part;       // -1: whole tile; else index of this K-part
  int tail;       // index of the tile among the split tiles
};

// Tile t of a tiles_m x tiles_n grid: column panels of kPanel tiles, all row tiles of a panel before
// the next panel. The tiles in flight at any time then share a few B panels and sweep A, so the
// set that has to stay in L2 between rounds is A (small) instead of all of B.
__device__ __forceinline__ void place_in_panels(int t, int tiles_m, int tiles_n, int* mt, int* nt) {
  constexpr int kPanel = KSB_FP8_PANEL;
  const int per_panel = kPanel * tiles_m;
  const int panel = t / per_panel;
  const int r = t - panel * per_panel;
  const int width = (tiles_n - panel * kPanel) < kPanel ? (tiles_n - panel * kPanel) : kPanel;
  *mt = r / width;
  *nt = panel * kPanel + (r - *mt * width);
}

// The K-split that a CTA goes by: Params' of a dense problem; a grouped one's tiles are whole, their number is
// known on the device only.
struct Split {
  int from, items, s;
};

// Parts that each of the `rem` tiles of a partial round is cut into along K: as many as the grid has
// CTAs for, at most eight (each part is one more partial to add up), and four K-blocks a part at least.
inline int split_parts(int grid, int rem, int nkb) {
  int s = grid / rem;
  if (s > 8) s = 8;
  while (s > 1 && nkb / s < 4) --s;
  return s;
}

template <int BN, bool GROUPED>
__device__ __forceinline__ bool locate_tile(const Params& p, const Split& sp, uint32_t tables, int t, TileCoord* tc) {
  tc->kb0 = 0;
  tc->kb1 = p.nkb;
  tc->part = -1;
  tc->tail = 0;
  if (!GROUPED && t >= sp.from) {
    const int r = t - sp.from;
    tc->tail = r / sp.s;
    tc->part = r - tc->tail * sp.s;
    tc->kb0 = (tc->part * p.nkb) / sp.s;
    tc->kb1 = ((tc->part + 1) * p.nkb) / sp.s;
    t = sp.from + tc->tail;
  }
  if constexpr (!GROUPED) {
    if (t >= p.tiles_m * p.tiles_n) return false;
    int mt, nt;
    place_in_panels(t, p.tiles_m, p.tiles_n, &mt, &nt);
    tc->expert = 0;
    tc->row0 = mt * kBM;
    tc->row_end = p.m;
    tc->n0 = nt * BN;
    return true;
  } else {
    // tables: row tiles before an expert | its first row | its end row
    const auto prefix = [&](int e) { return ld_shared_s32(tables + 4 * e); };
    const int total_mt = prefix(p.num_experts);
    if (t >= total_mt * p.tiles_n) return false;
    const int mt = t / p.tiles_n;
    int lo = 0, hi = p.num_experts - 1;  // last e with prefix[e] <= mt
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prefix(mid) <= mt) lo = mid; else hi = mid - 1;
    }
    // The expert's tiles in panels, like a dense problem's: with all columns of one row tile before
    // the next row tile, the second row tile of an expert found its weights gone from L2 where the
    // expert's weight is larger (K=4096, N=28672 in 16 bits: 235 MB) and read them from HBM again.
    const int first = prefix(lo);
    int em, en;
    place_in_panels(t - first * p.tiles_n, prefix(lo + 1) - first, p.tiles_n, &em, &en);
    tc->expert = lo;
    tc->row0 = ld_shared_s32(tables + 4 * (kMaxExperts + 1 + lo)) + em * kBM;
    tc->row_end = ld_shared_s32(tables + 4 * (2 * (kMaxExperts + 1) + lo));
    tc->n0 = en * BN;
    return true;
  }
}

// Work items of a CTA in the order it processes them: its K-part of a split tile first (if
// it has one), then whole tiles blockIdx.x, blockIdx.x + gridDim.x, ...
struct ItemWalk {
  int n;
  __device__ explicit ItemWalk(const Split& sp)
      : n((sp.s > 1 && static_cast<int>(blockIdx.x) < sp.items) ? -1 : 0) {}
  template <int BN, bool GROUPED>
  __device__ __forceinline__ bool next(const Params& p, const Split& sp, uint32_t tables, TileCoord* tc) {
    const int t = n < 0 ? sp.from + static_cast<int>(blockIdx.x)
                        : static_cast<int>(blockIdx.x) + n * static_cast<int>(gridDim.x);
    if (n >= 0 && t >= sp.from) return false;
    ++n;
    return locate_tile<BN, GROUPED>(p, sp, tables, t, tc);
  }
};

static_assert(Cfg<256>::smem_bytes(false) <= 232448 && Cfg<256>::smem_bytes(true) <= 232448 &&
                  Cfg<128>::smem_bytes(false) <= 232448 && Cfg<128>::smem_bytes(true) <= 232448,
              "shared memory layout exceeds the 227 KB a CTA can opt in to");
static_assert(128 * Cfg<256>::kRegsIssue + (Cfg<256>::kThreads - 128) * Cfg<256>::kRegsEpi <=
                  Cfg<256>::kThreads * ((65536 / Cfg<256>::kThreads) & ~7),
              "setmaxnreg budgets exceed the register pool the CTA is launched with");

// Four adjacent outputs, rounded once; `valid` of them lie inside the row.
template <typename OutT>
__device__ __forceinline__ void store_4(OutT* dst, const float4& v, bool vec_ok, int valid) {
  const float v4[4] = {v.x, v.y, v.z, v.w};
  if (vec_ok && valid >= 4) {
    if constexpr (std::is_same<OutT, float>::value) {
      *reinterpret_cast<float4*>(dst) = v;
    } else {
      OutT o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = from_f32<OutT>(v4[j]);
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < valid) dst[j] = from_f32<OutT>(v4[j]);
  }
}

// MODE 0: block-scaled FP8 (a partial per K-block, promoted in registers).
// MODE 1: FP8 with one scale per row of A and one per column of B: the whole K range
//         accumulates in tensor memory, the epilogue runs once per tile.
// MODE 2: the same with int8 operands (kind::i8, int32 accumulators) and an optional bias.
// MODE 3: f16 / bf16 operands (kind::f16), no scales: a K-block is 64 elements (the same 128
//         bytes per row), B stored [K,N] is loaded in 64-column atoms. The unscaled grouped GEMM.
template <int BN, bool NT, bool GROUPED, typename OutT, int MODE = 0>
__global__ void __launch_bounds__(Cfg<BN>::kThreads, 1)
fp8_blockwise_umma_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_a32,
                          const __grid_constant__ CUtensorMap tm_b,
                          const __grid_constant__ Params p) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  // Shared memory, from a 1024-byte boundary (for the 128 B swizzle): ring | store staging | full[S] | empty[S] |
  // tmem_empty[B] | acc_full[B] | slot_empty[] | tmem slot | abort flag | slots | tiles | grouped: tables.
  // Every role starts from a base of its own (base_of) and adds these: addresses that all roles share would
  // each take a register through all of them.
  constexpr uint32_t kStaging = C::kStages * C::kStageBytes;
  constexpr uint32_t kBarFull = kStaging + C::kStagingBytes;
  constexpr uint32_t kBarEmpty = kBarFull + 8 * C::kStages;
  constexpr uint32_t kBarTempty = kBarEmpty + 8 * C::kStages;
  constexpr uint32_t kBarAcc = kBarTempty + 8 * C::kAccBufs;   // MODE 1 / 2 / 3: a tile's accumulator is complete
  constexpr uint32_t kBarSempty = kBarAcc + 8 * C::kAccBufs;
  constexpr uint32_t kTmemSlot = kBarSempty + 8 * C::kSlots;
  constexpr uint32_t kSlotsAt = kBarFull + C::kCtrlBytes;
  constexpr uint32_t kTilesAt = kSlotsAt + C::kSlots * C::kSlotBytes;
  constexpr uint32_t kTables = kSlotsAt + C::kSchedBytes;
  static_assert(kTmemSlot + 8 <= kSlotsAt, "control block");
  // The barrier on which the epilogue waits also counts the arrival of the schedule's warp, whose lead, the
  // slots in use, is therefore no more than that barrier's turns: stages in MODE 0, accumulators otherwise.
  constexpr uint32_t kSlots = MODE == 0 ? C::kSlots : C::kAccBufs;
  static_assert(C::kSlots <= C::kStages && C::kAccBufs <= C::kSlots, "lead of the schedule");
  const auto base_of = [&]() {
    uint32_t b = (smem_u32(smem_raw) + 1023u) & ~1023u;
    asm volatile("" : "+r"(b));
    return b;
  };
  constexpr uint32_t kTilesTotal = kTmemSlot + 16;   // grouped: the number of tiles
  static_assert(kTilesTotal + 4 <= kSlotsAt, "control block");
  const auto split_of = [&](uint32_t sm) {
    return GROUPED ? Split{ld_shared_s32(sm + kTilesTotal), 0, 1}
                   : Split{p.split_from, p.split_items, p.split_s};
  };
  const auto wait_ctx = [&](uint32_t sm) { return WaitCtx{sm + kTmemSlot + 4, p.fault_word}; };
  uint8_t* const smem = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kTmemSlot);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    const uint32_t sm = base_of();
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(sm + kBarFull + 8 * s, 1);
      mbar_init(sm + kBarEmpty + 8 * s, MODE == 0 ? 2 : 1);   // commit; MODE 0: and the K-block's scales
    }
    for (int b = 0; b < C::kAccBufs; ++b) {
      mbar_init(sm + kBarTempty + 8 * b, C::kEpiWarps);
      mbar_init(sm + kBarAcc + 8 * b, 2);   // commit and the tile's place
    }
    for (int q = 0; q < C::kSlots; ++q) {
      mbar_init(sm + kBarSempty + 8 * q, C::kEpiWarps);
    }
    *abort_flag = 0u;
    fence_barrier_init();
    prefetch_tensormap(&tm_a);
    prefetch_tensormap(&tm_a32);
    prefetch_tensormap(&tm_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::kTmemCols);
    tmem_relinquish();
  }
  grid_dependency_wait();   // nothing before this touches memory that the kernel before may still write or read
  if constexpr (GROUPED) {
    // offs[e] = first row of expert e; with the masked layout the rows of an expert end at
    // offs[e] + masked_m[e] instead of at offs[e + 1] (ends[] holds either)
    int* prefix = reinterpret_cast<int*>(smem + kTables);
    int* offs = prefix + (kMaxExperts + 1);
    int* ends = offs + (kMaxExperts + 1);
    for (int e = threadIdx.x; e <= p.num_experts; e += blockDim.x) {
      if (p.masked_m != nullptr) {
        offs[e] = e * p.max_m;
        if (e < p.num_experts) {
          int mm = p.masked_m[e];
          mm = mm < 0 ? 0 : (mm > p.max_m ? p.max_m : mm);
          ends[e] = e * p.max_m + mm;
        }
      } else {
        offs[e] = p.offsets[e];
        if (e < p.num_experts) ends[e] = p.offsets[e + 1];
      }
    }
    __syncthreads();
    if (warp == 0) {
      int run = 0;
      for (int e0 = 0; e0 < p.num_experts; e0 += 32) {
        const int e = e0 + lane;
        const int rows = e < p.num_experts ? ends[e] - offs[e] : 0;
        const int tiles = rows > 0 ? (rows + kBM - 1) / kBM : 0;
        int inc = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        if (e < p.num_experts) prefix[e] = run + inc - tiles;
        run += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) {
        prefix[p.num_experts] = run;
        // (worked out by every role for itself, the product costs the 40-register warps spills)
        *reinterpret_cast<int*>(smem + kTilesTotal) = run * p.tiles_n;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if constexpr (C::kRebalanceRegs) setmaxnreg_dec<C::kRegsIssue>();
    const uint32_t sm = base_of();
    uint32_t it = 0;
    bool ok = true;
    TileCoord tc;
    const Split sp = split_of(sm);
    for (ItemWalk walk(sp); ok && walk.template next<BN, GROUPED>(p, sp, sm + kTables, &tc);) {
      // A tile of up to 32 rows takes a box of 32: the rows behind its end (of no matrix, or of the next
      // expert) stay away, and what the MMAs read there goes into rows that are not stored. M=16, N=14336:
      // K=7168 33.7 -> 25.4 us, K=4096 19.8 -> 17.2 (64 rows took 25.6 and 17.2 already); decode of 48 tokens
      // over 64 experts 251 -> 242. Up to three such boxes for 33 to 96 rows were slower than one of 128
      // (8 experts, K=14336, N=4096, 16 bits 204 -> 211 us), so more rows keep that.
      const bool few = tc.row_end - tc.row0 <= 32;
      for (int kb = tc.kb0; kb < tc.kb1; ++kb, ++it) {
        const uint32_t s = it % C::kStages;
        const uint32_t ph = (it / C::kStages) & 1u;
        if (!mbar_wait(wait_ctx(sm), sm + kBarEmpty + 8 * s, ph ^ 1u, 0x100u + s)) { ok = false; break; }
        {
          const uint32_t full = sm + kBarFull + 8 * s;
          const uint32_t a_dst = sm + s * C::kStageBytes;
          const uint32_t b_dst = a_dst + C::kABytes;
          if (few) {
            mbar_arrive_expect_tx_elect(full, C::kBBytes + 32 * kBK);
            tma_load_2d_elect(a_dst, &tm_a32, full, kb * kBK, tc.row0);
          } else {
            mbar_arrive_expect_tx_elect(full, C::kStageBytes);
            tma_load_2d_elect(a_dst, &tm_a, full, kb * kBK, tc.row0);
          }
          if constexpr (NT) {
            tma_load_3d_elect(b_dst, &tm_b, full, kb * kBK, tc.n0, tc.expert);
          } else if constexpr (MODE == 3) {
            // the map sees B as bytes: 64 columns of 16 bits = one 128-byte atom, 64 k-rows per K-block
#pragma unroll
            for (int h = 0; h < BN / 64; ++h)
              tma_load_3d_elect(b_dst + h * (64 * 128), &tm_b, full, 2 * tc.n0 + h * 128, kb * 64, tc.expert);
          } else {
#pragma unroll
            for (int h = 0; h < BN / 128; ++h)
              tma_load_3d_elect(b_dst + h * (128 * kBK), &tm_b, full, tc.n0 + h * 128, kb * kBK, tc.expert);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    if constexpr (C::kRebalanceRegs) setmaxnreg_dec<C::kRegsIssue>();
    const uint32_t sm = base_of();
    uint32_t it = 0;
    uint32_t tile_n = 0;   // MODE 1 / 2: tiles so far (one accumulator buffer per tile)
    bool ok = true;
    // what it needs of the walk is the number of K-blocks: a part of a split tile first, then whole tiles
    const Split sp = split_of(sm);
    int items = sp.from;
    items = (items - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    int nk = p.nkb;
    if (sp.s > 1 && static_cast<int>(blockIdx.x) < sp.items) {
      const int part = static_cast<int>(blockIdx.x) % sp.s;
      nk = ((part + 1) * p.nkb) / sp.s - (part * p.nkb) / sp.s;
      ++items;
    }
    for (; ok && items > 0; --items, nk = p.nkb) {
      if constexpr (MODE != 0) {
        const uint32_t tbuf = tile_n % C::kAccBufs, tph = (tile_n / C::kAccBufs) & 1u;
        if (!mbar_wait(wait_ctx(sm), sm + kBarTempty + 8 * tbuf, tph ^ 1u, 0x200u + tbuf)) { ok = false; break; }
      }
      for (int kb = 0; kb < nk; ++kb, ++it) {
        const uint32_t s = it % C::kStages;
        const uint32_t ph = (it / C::kStages) & 1u;
        const uint32_t buf = MODE != 0 ? tile_n % C::kAccBufs : it % C::kAccBufs;
        // A and (NT) B are K-major: 8-row groups 1024 B apart, a K step of 32
        // elements is 32 B inside the swizzle atom. B stored [K,N] is MN-major:
        // 128-column atoms 16 KB apart, 8-k groups 1024 B apart, a K step of 32
        // rows is 32 * 128 B.
        // (16-bit operands, MODE 3: the same bytes per instruction, 16 elements; an MN-major
        // atom is 64 columns x 64 k-rows = 8 KB and a K step of 16 rows is 16 * 128 B)
        const uint32_t a_src = sm + s * C::kStageBytes;
        const uint32_t b_src = a_src + C::kABytes;
        const uint32_t d_tmem = tmem_base + buf * BN;
        uint64_t a_desc[kBK / 32], b_desc[kBK / 32];
#pragma unroll
        for (int kk = 0; kk < kBK / 32; ++kk) {
          a_desc[kk] = umma_smem_desc_sw128(a_src + kk * 32, 16, 1024);
          b_desc[kk] = NT ? umma_smem_desc_sw128(b_src + kk * 32, 16, 1024)
                     : MODE == 3 ? umma_smem_desc_sw128(b_src + kk * 16 * 128, 64 * 128, 1024)
                                 : umma_smem_desc_sw128(b_src + kk * 32 * 128, 128 * kBK, 1024);
        }
        // The operands are tested first: they are there long before the accumulator buffer is handed
        // back, and even a test that succeeds takes ~100 cycles, which in the other order lay between the
        // release of the buffer and the MMAs that it lets start.
        if (!mbar_wait(wait_ctx(sm), sm + kBarFull + 8 * s, ph, 0x300u + s)) { ok = false; break; }
        if constexpr (MODE == 0) {
          const uint32_t aph = (it / C::kAccBufs) & 1u;
          if (!mbar_wait(wait_ctx(sm), sm + kBarTempty + 8 * buf, aph ^ 1u, 0x200u + buf)) { ok = false; break; }
        }
        tc_fence_after_sync();
        {
          // all 32 lanes run this code; each instruction elects its one issuing lane
#pragma unroll
          for (int kk = 0; kk < kBK / 32; ++kk) {
            const uint32_t accumulate = (kk > 0 || (MODE != 0 && kb > 0)) ? 1u : 0u;
            if constexpr (MODE == 2) umma_i8_elect(d_tmem, a_desc[kk], b_desc[kk], p.idesc, accumulate);
            else if constexpr (MODE == 3) umma_f16_elect(d_tmem, a_desc[kk], b_desc[kk], p.idesc, accumulate);
            else umma_f8f6f4_elect(d_tmem, a_desc[kk], b_desc[kk], p.idesc, accumulate);
          }
          tc_commit_elect(sm + kBarEmpty + 8 * s);
          if constexpr (MODE != 0) {
            if (kb == nk - 1) tc_commit_elect(sm + kBarAcc + 8 * buf);
          }
        }
      }
      ++tile_n;
    }
  } else if (warp >= 4) {
    // -------------------------------- epilogue --------------------------------
    if constexpr (C::kRebalanceRegs) setmaxnreg_inc<C::kRegsEpi>();
    const int quarter = warp & 3;         // TMEM lane quarter this warp can address
    const int slice = (warp - 4) >> 2;    // which kEpiCols-wide column slice of the tile
    constexpr int EC = C::kEpiCols;
    const int row_in_tile = quarter * 32 + lane;
    OutT* out = static_cast<OutT*>(p.out);
    uint32_t it = 0;       // slots read so far: K-blocks in MODE 0, tiles otherwise
    uint32_t tile_n = 0;
    bool ok = true;
    const uint32_t my_scale = (slice * kBM + row_in_tile) * 4;   // within a slot
    while (true) {
      const uint32_t sm = base_of();
      // the tile's first K-block, or (MODE 1, 2, 3) all of it, and its place
      const uint32_t turns = MODE == 0 ? C::kStages : C::kAccBufs;
      const uint32_t done = (MODE == 0 ? sm + kBarEmpty : sm + kBarAcc) + 8 * (it % turns);
      if (!(MODE == 0 ? mbar_wait_hinted(wait_ctx(sm), done, (it / turns) & 1u, 0x400u + it % turns, 50u)
                      : mbar_wait_long(wait_ctx(sm), done, (it / turns) & 1u, 0x400u + it % turns))) {
        ok = false;
        break;
      }
      const uint32_t tile_at = sm + kTilesAt + (tile_n++ % C::kTileSlots) * C::kTileBytes;
      const int nk = ld_shared_s32(tile_at);
      if (nk == 0) break;   // no more work

      float2 acc[EC / 2];
#pragma unroll
      for (int i = 0; i < EC / 2; ++i) acc[i] = make_float2(0.f, 0.f);

      if constexpr (MODE != 0) {
        // the tile's accumulator is complete: scale by a_scale[row] * b_scale[col] (and add
        // the bias) on the way out of tensor memory, as kernels/src/gemm/gemm_fp8.cu:147-153
        // and gemm_w8a8.cu:134-141 of the reference do
        const uint32_t tbuf = it % C::kAccBufs;
        tc_fence_after_sync();
        const int row = ld_shared_s32(tile_at + 4) + row_in_tile;
        const bool row_ok = row < ld_shared_s32(tile_at + 8);
        const int col0 = ld_shared_s32(tile_at + 12) + slice * EC;
        float a_sc = 1.f, b_one = 1.f;
        if constexpr (MODE != 3) {
          a_sc = (p.a_per_row && row_ok) ? __ldg(p.a_scale + row) : __ldg(p.a_scale);
          b_one = __ldg(p.b_scale);
        }
        const OutT* bias = static_cast<const OutT*>(p.bias);
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + tbuf * BN + slice * EC;
#pragma unroll
        for (int c = 0; c < EC / 16; ++c) {
          uint32_t r[16];
          tmem_ld(taddr + c * 16, r);
          tmem_wait_ld(r);
          if (c == EC / 16 - 1) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(sm + kBarTempty + 8 * tbuf);
              mbar_arrive(sm + kBarSempty + 8 * (it % kSlots));
            }
          }
          float v2[16];
          // (the columns' numbers are worked out 16 at a time: all at once they are spilled)
          int colc = col0 + c * 16;
          asm volatile("" : "+r"(colc));
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int col = colc + j;
            const bool col_ok = col < p.n;
            const float raw = MODE == 2 ? static_cast<float>(static_cast<int32_t>(r[j])) : __uint_as_float(r[j]);
            float v = raw;
            if constexpr (MODE != 3) {
              const float b_sc = (p.b_per_col && col_ok) ? __ldg(p.b_scale + col) : b_one;
              v = __fmul_rn(__fmul_rn(raw, a_sc), b_sc);
              if (bias != nullptr && col_ok) v = __fadd_rn(v, to_f32<OutT>(bias[col]));
            }
            v2[j] = v;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[c * 8 + j] = make_float2(v2[2 * j], v2[2 * j + 1]);
        }
        ++it;
      }

      // The promotion: one K-block per pass of a rolled loop, its scale one shared-memory load.
      if constexpr (MODE == 0) {
        constexpr int CW = 16;   // TMEM columns per load
        const uint32_t tquarter = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + slice * EC;
        int kb = nk;
#pragma unroll 1
        while (true) {
          // (every address from one base: kept apart they would take registers that the accumulators need)
          const uint32_t sm = base_of();
          tc_fence_after_sync();
          const uint32_t buf = it % C::kAccBufs, slot = it % kSlots;
          const uint32_t taddr = tquarter + buf * BN;
          uint32_t r0[CW], r1[CW];
          tmem_ld(taddr, r0);
          const float sc = ld_shared_f32(sm + kSlotsAt + slot * C::kSlotBytes + my_scale);
          const float2 scale2 = make_float2(sc, sc);
#pragma unroll
          for (int c = 0; c < EC / CW; ++c) {
            if (c & 1) tmem_wait_ld(r1);
            else tmem_wait_ld(r0);
            if (c < EC / CW - 1) {
              if (c & 1) tmem_ld(taddr + (c + 1) * CW, r0);
              else tmem_ld(taddr + (c + 1) * CW, r1);
            } else {
              // every column of this warp's slice is in registers: hand the buffer back
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) {
                mbar_arrive(sm + kBarTempty + 8 * buf);
                mbar_arrive(sm + kBarSempty + 8 * slot);
              }
            }
#pragma unroll
            for (int j = 0; j < CW / 2; ++j) {
              const float lo = __uint_as_float((c & 1) ? r1[2 * j] : r0[2 * j]);
              const float hi = __uint_as_float((c & 1) ? r1[2 * j + 1] : r0[2 * j + 1]);
              ffma2(acc[c * (CW / 2) + j], lo, hi, scale2);
            }
          }
          ++it;
          if (--kb == 0) break;
          // One tcgen05.commit per K-block serves both consumers: the barrier that hands the
          // shared-memory stage back to the producer also tells the epilogue that the
          // accumulator is complete (each extra commit costs the tensor core ~50 idle cycles).
          // short suspend hint: these warps are the critical path of every K-block, and a
          // waiter parked for the default period is resumed later than one that re-polls
          if (!mbar_wait_hinted(wait_ctx(sm), sm + kBarEmpty + 8 * (it % C::kStages), (it / C::kStages) & 1u,
                                0x400u + it % C::kStages, 50u)) {
            ok = false;
            break;
          }
        }
      }
      // (the rest of the tile's place is not held in registers over the K loop)
      const uint4 t0 = ld_shared_v4(tile_at);
      const uint4 t1 = ld_shared_v4(tile_at + 16);
      struct { int row0, row_end, n0, part, tail, parts; } tc;
      tc.row0 = static_cast<int>(t0.y);
      tc.row_end = static_cast<int>(t0.z);
      tc.n0 = static_cast<int>(t0.w);
      tc.part = static_cast<int>(t1.x);
      tc.tail = static_cast<int>(t1.y);
      tc.parts = static_cast<int>(t1.z);
      const int row = tc.row0 + row_in_tile;
      const bool row_ok = row < tc.row_end;
      const int col0 = tc.n0 + slice * EC;
      bool stored = false;
      if constexpr (!GROUPED) {
        if (ok && tc.part >= 0 && p.cluster_s > 1) {
          // One K-part of a tile that the cluster shares: rows of BN + 4 floats (the padding
          // keeps the 16-byte stores of eight neighbouring lanes on different banks).
          if (row_ok) {
            const uint32_t dst = sm + (row_in_tile * (BN + 4) + slice * EC) * 4;
#pragma unroll
            for (int c4 = 0; c4 < EC / 4; ++c4)
              st_shared_v4(dst + c4 * 16, __float_as_uint(acc[2 * c4].x), __float_as_uint(acc[2 * c4].y),
                           __float_as_uint(acc[2 * c4 + 1].x), __float_as_uint(acc[2 * c4 + 1].y));
          }
          stored = true;
        }
      }
      if constexpr (!GROUPED) {
        if (ok && !stored && tc.part >= 0) {
          // One K-part of a split tile. The warp's 32 x EC partial goes to its slot (16 bytes per lane and column
          // chunk, chunks 512 B apart: every store of the warp is one contiguous 512-byte piece); split_reduce_kernel
          // adds the parts up afterwards, on all SMs (M=2500, N=2000, K=4096 35.0 us, 44.0 with the sums in here).
          // Rows that do not exist stay away, 32 at a time.
          stored = true;
          if (tc.row0 + quarter * 32 < tc.row_end) {
            constexpr int kChunks = EC / 4;      // float4 chunks per lane
            int ew = warp - 4;
            asm volatile("" : "+r"(ew));   // (as below: nothing of this is to be worked out ahead)
            float4* mine = p.split_slots + ((static_cast<size_t>(tc.tail) * tc.parts + tc.part) * C::kEpiWarps + ew) * (kChunks * 32) + lane;
#pragma unroll
            for (int c4 = 0; c4 < kChunks; ++c4)
              __stcg(mine + c4 * 32, make_float4(acc[2 * c4].x, acc[2 * c4].y, acc[2 * c4 + 1].x, acc[2 * c4 + 1].y));
          }
        }
      }
      if (ok && !stored && p.vec_store) {
        // The warp's 32 x EC block leaves in pieces of 32 rows x 64 bytes: a lane writes its row to
        // shared memory (16-byte chunks swizzled so that neighbouring lanes hit different banks), then
        // four lanes read a row and store it. (By TMA store every piece waited for the one before to be
        // read; from the lanes' own rows, as grouped problems had it, every 16-byte store touched 32 lines.)
        constexpr int kPieceCols = C::kPieceBytes / static_cast<int>(sizeof(OutT));
        constexpr int kChunkCols = 16 / static_cast<int>(sizeof(OutT));
        constexpr int kChunks = C::kPieceBytes / 16;
        constexpr int kRows = 32 / kChunks;   // rows that the warp reads at a time
        static_assert(kChunks == 4, "the swizzle");
        // (the compiler is kept from working out the addresses below once for all tiles: they would take the K
        // loop's registers)
        int ln = lane;
        asm volatile("" : "+r"(ln));
        const uint32_t my_stage = sm + kStaging + (warp - 4) * (32 * C::kPieceBytes);   // aligned to its size
        // chunk j of row r lies at r * 64 + 16 * (j ^ ((r >> 1) & 3))
        const uint32_t w_base = my_stage + ln * C::kPieceBytes + (((ln >> 1) & 3) << 4);
        const int r0 = ln / kChunks, cj = ln % kChunks;   // this lane reads chunk cj of rows r0, r0 + 8, ...
        const uint32_t r_base = my_stage + r0 * C::kPieceBytes + ((cj ^ ((r0 >> 1) & 3)) << 4);
        OutT* dst = out;
        int dst_row = tc.row0 + quarter * 32;
        if constexpr (!GROUPED) {
          if (p.rows_per_part > 0) {   // a tile lies inside one part: rows_per_part is a multiple of its height
            const int part = tc.row0 / p.rows_per_part;
            dst = static_cast<OutT*>(p.out_parts[part]);
            dst_row -= part * p.rows_per_part;
          }
        }
        const int rows = tc.row_end - (tc.row0 + quarter * 32);   // of this warp's 32 that exist
        dst += static_cast<size_t>(dst_row + r0) * p.n + col0 + cj * kChunkCols;
#pragma unroll
        for (int pc = 0; pc < EC / kPieceCols; ++pc) {
          if (col0 + pc * kPieceCols >= p.n || rows <= 0) break;   // warp-uniform
          __syncwarp();   // the piece before has been read
#pragma unroll
          for (int j = 0; j < kChunks; ++j) {
            const uint4 w = pack_16_bytes<OutT>(acc, pc * kPieceCols + j * kChunkCols);
            st_shared_v4(w_base ^ (j << 4), w.x, w.y, w.z, w.w);
          }
          __syncwarp();
          const bool col_ok = col0 + pc * kPieceCols + cj * kChunkCols < p.n;   // rows are whole chunks here
#pragma unroll
          for (int i = 0; i < kChunks; ++i) {
            const uint4 w = ld_shared_v4(r_base + i * kRows * C::kPieceBytes);
            if (col_ok && i * kRows + r0 < rows)
              *reinterpret_cast<uint4*>(dst + static_cast<size_t>(i * kRows) * p.n + pc * kPieceCols) = w;
          }
        }
        stored = true;
      }
      if (ok && row_ok && !stored) {
        OutT* dst = out + static_cast<size_t>(row) * p.n + col0;
#pragma unroll
        for (int c = 0; c < EC / 16; ++c) {
          const int valid = p.n - (col0 + c * 16);
          float v[16];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            v[2 * j] = acc[c * 8 + j].x;
            v[2 * j + 1] = acc[c * 8 + j].y;
          }
          if (valid > 0) store_16<OutT>(dst + c * 16, v, p.vec_store != 0, valid);
        }
      }
      if (!ok) break;
    }
  } else {
    // -------------------------- schedule and scales ---------------------------
    // Warps 2 and 3 walk the tiles ahead of the epilogue and hand it, K-block by K-block in turn, a slot
    // with the scales of the block's 128 rows and of the two column slices, and the tile (MODE 1, 2, 3: one
    // slot per tile, no scales). The epilogue warps then neither divide nor search for their next tile, nor
    // wait for a load from L2 or HBM between two tiles, and read a scale with one shared-memory load where
    // each of them had a load over 32 cache lines per K-block.
    if constexpr (C::kRebalanceRegs) setmaxnreg_dec<C::kRegsIssue>();
    const uint32_t sm = base_of();
    const uint32_t mine = static_cast<uint32_t>(warp - 2);
    uint32_t it = 0, tile_n = 0;
    bool ok = true;
    TileCoord tc;
    const Split sp = split_of(sm);
    for (ItemWalk walk(sp); ok && walk.template next<BN, GROUPED>(p, sp, sm + kTables, &tc);) {
      const int nk = MODE == 0 ? tc.kb1 - tc.kb0 : 1;
      const int first = static_cast<int>((it ^ mine) & 1u);   // this warp's first K-block of the tile
      const float* ap = nullptr;   // row 0 of the tile, and the other rows' distance from there
      int off[4] = {};
      const float* bp = nullptr;
      if constexpr (MODE == 0) {
        const int64_t kb = tc.kb0 + first;
        ap = p.a_scale + tc.row0 * p.as_row_stride + kb * p.as_kb_stride;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = i * 32 + lane, last = tc.row_end - 1 - tc.row0;
          off[i] = (r < last ? r : last) * static_cast<int>(p.as_row_stride);
        }
        int nb = (tc.n0 + ((lane >> 4) & 1) * C::kEpiCols) >> 7;   // lanes 0-15 the first slice, 16-31 the second
        if (nb > p.nnb - 1) nb = p.nnb - 1;
        bp = p.b_scale + static_cast<int64_t>(tc.expert) * p.nkb * p.nnb + (NT ? nb * static_cast<int64_t>(p.nkb) + kb : kb * p.nnb + nb);
      }
      for (int kb = first; kb < nk; kb += 2) {
        const uint32_t n = it + static_cast<uint32_t>(kb);
        const uint32_t slot = n % kSlots;
        const uint32_t base = sm + kSlotsAt + slot * C::kSlotBytes;
        float a[4], b = 0.f;
        if constexpr (MODE == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i] = ld_global_nc_f32(ap + off[i]);
          ap += 2 * p.as_kb_stride;
          b = ld_global_nc_f32(bp);
          bp += NT ? 2 : 2 * static_cast<int64_t>(p.nnb);
        }
        if (!mbar_wait(wait_ctx(sm), sm + kBarSempty + 8 * slot, ((n / kSlots) & 1u) ^ 1u, 0x600u + slot)) { ok = false; break; }
        if constexpr (MODE == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            st_shared_f32(base + (i * 32 + lane) * 4, a[i] * __shfl_sync(0xffffffffu, b, 0));
            st_shared_f32(base + (kBM + i * 32 + lane) * 4, a[i] * __shfl_sync(0xffffffffu, b, 16));
          }
        }
        if (kb == 0 && lane == 2) {
          const uint32_t at = sm + kTilesAt + (tile_n % C::kTileSlots) * C::kTileBytes;
          st_shared_v4(at, nk, tc.row0, tc.row_end, tc.n0);
          st_shared_v4(at + 16, tc.part, tc.tail, sp.s, 0);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(MODE == 0 ? sm + kBarEmpty + 8 * (n % C::kStages) : sm + kBarAcc + 8 * (n % C::kAccBufs));
      }
      it += static_cast<uint32_t>(nk);
      ++tile_n;
    }
    if (ok && ((it ^ mine) & 1u) == 0u) {   // the last slot says that there is no more
      const uint32_t slot = it % kSlots;
      if (mbar_wait(wait_ctx(sm), sm + kBarSempty + 8 * slot, ((it / kSlots) & 1u) ^ 1u, 0x600u + slot)) {
        if (lane == 0) {
          st_shared_v4(sm + kTilesAt + (tile_n % C::kTileSlots) * C::kTileBytes, 0, 0, 0, 0);
          const uint32_t bar = MODE == 0 ? sm + kBarEmpty + 8 * (it % C::kStages) : sm + kBarAcc + 8 * (it % C::kAccBufs);
          mbar_arrive(bar);   // twice: there is no commit
          mbar_arrive(bar);
        }
      }
    }
  }

  if constexpr (!GROUPED && MODE == 0) {
    static_assert(kBM * (BN + 4) * 4 <= C::kStages * C::kStageBytes, "the partial tile fits the ring");
    if (p.cluster_s > 1) {
      __syncwarp();
      cluster_sync();   // every CTA's partial is in its shared memory
      if (warp >= 4) {
        const uint32_t sm = base_of();
        // this CTA's share of the tile, in units of four columns
        TileCoord tc;
        locate_tile<BN, GROUPED>(p, split_of(sm), sm + kTables, static_cast<int>(blockIdx.x), &tc);
        const int rows = tc.row_end - tc.row0 < kBM ? tc.row_end - tc.row0 : kBM;
        const int total = rows * (BN / 4);
        const int begin = (tc.part * total) / p.cluster_s, end = ((tc.part + 1) * total) / p.cluster_s;
        for (int i = begin + static_cast<int>(threadIdx.x) - 128; i < end; i += C::kEpiWarps * 32) {
          const int r = i / (BN / 4), col = tc.n0 + (i % (BN / 4)) * 4;
          if (col >= p.n) continue;
          const uint32_t src = sm + (r * (BN + 4) + (i % (BN / 4)) * 4) * 4;
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int q = 0; q < p.cluster_s; ++q) {
            const float4 v = ld_shared_cluster_f4(cluster_map_shared(src, q));
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
          store_4<OutT>(static_cast<OutT*>(p.out) + static_cast<size_t>(tc.row0 + r) * p.n + col, sum,
                        p.vec_store != 0, p.n - col);
        }
      }
      __syncwarp();
      cluster_sync();   // nobody reads this CTA's shared memory any more
    }
  }

  // ------------------------------- teardown -------------------------------
  // Parts of a split round: the next kernel is split_reduce_kernel, which waits, and lines up from here on
  // (M=2500, N=2000, K=4096 37.3 -> 35.0 us).
  if (!GROUPED && p.split_slots != nullptr) grid_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    // A wait gave up: give copies and MMAs still in flight time to land
    // before shared memory and TMEM are released.
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// Sum of the K-parts of the split tiles: one thread per (tile, epilogue warp, column chunk,
// lane) reads its 16 bytes of every part in part order and writes four outputs.
template <int BN, typename OutT>
__global__ void __launch_bounds__(256)
split_reduce_kernel(OutT* __restrict__ out, const float4* __restrict__ slots, int split_from, int split_s, int tails,
                    int tiles_m, int tiles_n, int m, int n, int vec_ok) {
  using C = Cfg<BN>;
  grid_dependency_wait();
  constexpr int EC = C::kEpiCols;
  constexpr int kChunks = EC / 4;
  constexpr int kPerTile = C::kEpiWarps * kChunks * 32;   // float4 per (tile, part)
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= tails * kPerTile) return;
  const int tail = idx / kPerTile;
  const int r = idx - tail * kPerTile;
  const int ew = r / (kChunks * 32);
  const int c4 = (r / 32) % kChunks;
  const int lane = r & 31;
  // the tile's place in the output: the column-panel order of locate_tile
  int mt, nt;
  place_in_panels(split_from + tail, tiles_m, tiles_n, &mt, &nt);
  const int row = mt * kBM + (ew & 3) * 32 + lane;
  const int col = nt * BN + (ew >> 2) * EC + 4 * c4;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4* src = slots + static_cast<size_t>(tail) * split_s * kPerTile + r;
  for (int q = 0; q < split_s; ++q) {
    const float4 v = __ldcs(src + static_cast<size_t>(q) * kPerTile);
    sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
  }
  if (row >= m || col >= n) return;
  store_4<OutT>(out + static_cast<size_t>(row) * n + col, sum, vec_ok != 0, n - col);
}

// ------------------------------- host side --------------------------------
// Byte tensor of rank 2 or 3 (innermost first), 128-byte swizzled boxes.
bool encode_u8(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
               const uint32_t* box) {
  return tma_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, base, dims, strides_bytes, box,
                    CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int BN, bool NT, bool GROUPED, typename OutT, int MODE = 0>
ks_status_t launch_one(const Fp8GemmArgs& a, const CUtensorMap& tm_a, const CUtensorMap& tm_a32, const CUtensorMap& tm_b, Params p,
                       int grid, cudaStream_t stream) {
  using C = Cfg<BN>;
  auto kernel = fp8_blockwise_umma_kernel<BN, NT, GROUPED, OutT, MODE>;
  static std::mutex mu;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
      cudaError_t e =
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes(GROUPED));
      if (e != cudaSuccess) return cuda_status(e, a.where);
      attr_done[dev] = true;
    }
  }
  if (a.num_out_parts > 0 && !p.vec_store)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, std::string(a.where) + ": the scattered output needs 16-byte aligned rows and parts");
  // A short problem is set up under the tail of the kernel before it (the quantizer, a gather), which saves 2-3 us:
  // M=2500, N=2000, K=4096 behind the quantizer 44.0 -> 40.8 us, 48 tokens over 64 experts 249 -> 240, M=4096,
  // N=K=7168 behind the norm 248 -> 245 (339 K-blocks per CTA). A long one loses 1 % that way (M=16384, N=8192, K=3584,
  // 775 K-blocks: 600 -> 609), so from 512 on it is launched the ordinary way. The GEMM does not let
  // its own successor begin early: with that the same four took 42.7, 245, 252 and 614.
  const int64_t tiles = p.tiles_n * (GROUPED ? (a.m + kBM - 1) / kBM + p.num_experts : static_cast<int64_t>(p.tiles_m));
  const bool is_short = tiles * p.nkb <= 512 * static_cast<int64_t>(sm_count());
  const cudaError_t e = launch_programmatic_cluster(kernel, grid, p.cluster_s, is_short, C::kThreads,
                                                    C::smem_bytes(GROUPED), stream, tm_a, tm_a32, tm_b, p);
  if (e != cudaSuccess) return cuda_status(e, a.where);
  if constexpr (!GROUPED) {
    if (p.split_slots != nullptr) {   // (a cluster adds its parts up itself)
      const int tails = p.split_items / p.split_s;
      const int work = tails * C::kEpiWarps * (C::kEpiCols / 4) * 32;
      launch_programmatic(split_reduce_kernel<BN, OutT>, (work + 255) / 256, 256, 0, stream,
          static_cast<OutT*>(p.out), p.split_slots, p.split_from, p.split_s, tails, p.tiles_m, p.tiles_n, p.m, p.n,
          p.vec_store);
    }
  }
  return cuda_status(cudaGetLastError(), a.where);
}

template <int BN, bool NT, bool GROUPED, int MODE = 0>
ks_status_t launch_out(const Fp8GemmArgs& a, const CUtensorMap& tm_a, const CUtensorMap& tm_a32, const CUtensorMap& tm_b, const Params& p,
                       int grid, cudaStream_t stream) {
  switch (a.out_dtype) {
    case KS_DTYPE_F32: return launch_one<BN, NT, GROUPED, float, MODE>(a, tm_a, tm_a32, tm_b, p, grid, stream);
    case KS_DTYPE_F16: return launch_one<BN, NT, GROUPED, __half, MODE>(a, tm_a, tm_a32, tm_b, p, grid, stream);
    default: return launch_one<BN, NT, GROUPED, __nv_bfloat16, MODE>(a, tm_a, tm_a32, tm_b, p, grid, stream);
  }
}

template <int BN>
ks_status_t launch_bn(const Fp8GemmArgs& a, const CUtensorMap& tm_a, const CUtensorMap& tm_a32, const CUtensorMap& tm_b, const Params& p,
                      int grid, cudaStream_t stream) {
  const bool grouped = a.offsets != nullptr || a.masked_m != nullptr;
  // the per-row / per-column scaled kernels exist for the reference's layout (B stored [K,N]), dense
  if (a.mode == 1) return launch_out<BN, false, false, 1>(a, tm_a, tm_a32, tm_b, p, grid, stream);
  if (a.mode == 2) return launch_out<BN, false, false, 2>(a, tm_a, tm_a32, tm_b, p, grid, stream);
  // 16-bit operands, B stored [K,N]: the output has the operands' type
  if (a.mode == 3) {
    if (a.out_dtype == KS_DTYPE_F16)
      return grouped ? launch_one<BN, false, true, __half, 3>(a, tm_a, tm_a32, tm_b, p, grid, stream)
                     : launch_one<BN, false, false, __half, 3>(a, tm_a, tm_a32, tm_b, p, grid, stream);
    return grouped ? launch_one<BN, false, true, __nv_bfloat16, 3>(a, tm_a, tm_a32, tm_b, p, grid, stream)
                   : launch_one<BN, false, false, __nv_bfloat16, 3>(a, tm_a, tm_a32, tm_b, p, grid, stream);
  }
  if (a.nt) return grouped ? launch_out<BN, true, true>(a, tm_a, tm_a32, tm_b, p, grid, stream)
                           : launch_out<BN, true, false>(a, tm_a, tm_a32, tm_b, p, grid, stream);
  return grouped ? launch_out<BN, false, true>(a, tm_a, tm_a32, tm_b, p, grid, stream)
                 : launch_out<BN, false, false>(a, tm_a, tm_a32, tm_b, p, grid, stream);
}

}  // namespace

bool fp8_blockwise_eligible(const Fp8GemmArgs& a) {
  if (a.mode == 0 && (a.block_n != 128 || a.block_k != 128)) return false;
  if ((a.mode == 1 || a.mode == 2) && (a.nt || a.offsets != nullptr || a.masked_m != nullptr)) return false;
  if (a.mode == 3) {
    // 16-bit operands: 16-byte row pitches of A [M,K] and B [K,N]
    if (a.nt || a.masked_m != nullptr || a.k % 8 != 0 || a.n % 8 != 0) return false;
    if (a.out_dtype != KS_DTYPE_F16 && a.out_dtype != KS_DTYPE_BF16) return false;
  } else {
    if (a.k % 16 != 0) return false;
    if (!a.nt && a.n % 16 != 0) return false;
  }
  if (!aligned16(a.a) || !aligned16(a.b)) return false;
  if (a.m > INT32_MAX / 2 || a.n > INT32_MAX / 2 || a.k > INT32_MAX / 2) return false;
  if ((a.offsets != nullptr || a.masked_m != nullptr) && (a.num_experts > kMaxExperts || a.num_experts < 1)) return false;
  if (a.masked_m != nullptr && (a.max_m < 1 || a.max_m * a.num_experts != a.m)) return false;
  return tma_available();
}

ks_status_t launch_fp8_blockwise(const Fp8GemmArgs& a, cudaStream_t stream) {
  const bool grouped = a.offsets != nullptr || a.masked_m != nullptr;
  const int experts = grouped ? a.num_experts : 1;
  const int sms = sm_count();
  const int64_t tiles_m_bound = grouped ? (a.m + kBM - 1) / kBM + experts : (a.m + kBM - 1) / kBM;
  // Tile width by estimated time: rounds of tiles over the SMs times the cost of a
  // K-block of that width (850 cycles for 128 x 256, 550 for 128 x 128, measured before warps 2 and 3 took over
  // scales and tiles; the wide loop takes ~727 since, and these figures and the 9000 and 14000 below, which
  // stand beside them, have not been fitted again). Wide tiles win
  // as soon as they do not need more rounds than narrow ones would save.
  // (grouped: by the bound of the row tiles. Their number is on the device only; by the number to expect,
  // max(experts hit, rows / 128 + experts / 2), even routings gained up to 30 %, but 54 of 432 measured shapes lost:
  // all rows to one expert up to 36 %, skewed routings 5-10, even ones up to 5.)
  const int64_t tiles256 = tiles_m_bound * ((a.n + 255) / 256);
  const int64_t tiles128 = tiles_m_bound * ((a.n + 127) / 128);
  // (with one scale per row and column nothing is promoted per K-block: the MMAs run back to
  // back, ~512 / ~300 cycles per K-block, and the wide tile wins whenever it needs no more rounds)
  const int64_t cost256 = ((tiles256 + sms - 1) / sms) * (a.mode == 0 ? 850 : 512);
  const int64_t cost128 = ((tiles128 + sms - 1) / sms) * (a.mode == 0 ? 550 : 300);
  int bn = (a.force_bn == 128 || a.force_bn == 256) ? a.force_bn : (cost256 <= cost128 ? 256 : 128);

  // Fewer tiles than SMs (dense block-scaled problems): cut every tile along K over a cluster of
  // S CTAs. Same unit of cost, and never less than the weight takes from HBM (~3500 bytes a cycle). Sharing
  // a tile costs ~9000 cycles by the shapes above and in the header: two cluster barriers, the
  // exchange of the partials, and a pipeline fill that fewer K-blocks pay for (M=94, N=11632, K=7040 is
  // better left to 91 unshared tiles of 128 columns). At least two K-blocks per CTA.
  int cluster_s = 1;
  if (!grouped && a.mode == 0 && a.force_split != 0 && a.num_out_parts == 0) {
    const int64_t nkb = (a.k + kBK - 1) / kBK;
    const int64_t hbm = a.n * a.k / 3500;
    int64_t best = INT64_MAX;
    for (int w = 256; w >= 128; w -= 128) {
      if ((a.force_bn == 128 || a.force_bn == 256) && a.force_bn != w) continue;
      const int64_t tiles = w == 256 ? tiles256 : tiles128;
      const int64_t per_kb = w == 256 ? 850 : 550;
      // full rounds of tiles, then the partial round: a whole round, or (see below) its tiles cut
      // along K over the idle SMs, plus the partials' way through memory and the reducing kernel:
      // 10000 to 16000 cycles by shapes where one width needs it and the other does not. Without
      // the second form 160 tiles of 256 columns counted as two rounds and lost to 320 of 128:
      // M=2500, N=2000, K=4096 42.0 -> 37.9 us; M=426, N=10528, K=15616 107.5 -> 91.1.
      const int64_t rem = tiles % sms;
      int64_t part = nkb;
      int64_t extra = 0;
      if (rem > 0 && tiles > sms) {
        const int64_t s = split_parts(sms, static_cast<int>(rem), static_cast<int>(nkb));
        if (s >= 2) {
          part = (nkb + s - 1) / s;
          extra = 14000;
        }
      }
      const int64_t chain = (tiles / sms * nkb + (rem > 0 ? part : 0)) * per_kb;
      const int64_t whole = (chain > hbm ? chain : hbm) + extra;
      if (whole < best) {
        best = whole;
        bn = w;
        cluster_s = 1;
      }
      for (int s = 2; s <= kMaxClusterSplit && tiles * s <= sms && nkb >= 2 * s; ++s) {
        if (cluster_capacity(s) < tiles) break;   // all clusters run at once
        const int64_t shared = (nkb + s - 1) / s * per_kb;
        const int64_t cost = (shared > hbm ? shared : hbm) + 9000;
        if (cost < best) {
          best = cost;
          bn = w;
          cluster_s = s;
        }
      }
    }
  }

  CUtensorMap tm_a, tm_a32, tm_b;
  // 16-bit operands (mode 3) are described to TMA as bytes: a row of A is 2K bytes, of B 2N
  const int64_t k_bytes = a.mode == 3 ? 2 * a.k : a.k;
  if (a.mode == 3) {
    const uint64_t dims[2] = {static_cast<uint64_t>(k_bytes), static_cast<uint64_t>(a.m)};
    const uint64_t str[1] = {static_cast<uint64_t>(k_bytes)};
    const uint32_t box[2] = {static_cast<uint32_t>(kBK), static_cast<uint32_t>(kBM)};
    const uint32_t box32[2] = {static_cast<uint32_t>(kBK), 32u};
    if (!encode_u8(&tm_a, a.a, 2, dims, str, box) || !encode_u8(&tm_a32, a.a, 2, dims, str, box32))
      KSB_FAIL(KS_ERROR_INTERNAL, std::string(a.where) + ": tensor map for A rejected");
    const uint64_t bdims[3] = {static_cast<uint64_t>(2 * a.n), static_cast<uint64_t>(a.k), static_cast<uint64_t>(experts)};
    const uint64_t bstr[2] = {static_cast<uint64_t>(2 * a.n), static_cast<uint64_t>(2 * a.n) * static_cast<uint64_t>(a.k)};
    const uint32_t bbox[3] = {128u, 64u, 1u};
    if (!encode_u8(&tm_b, a.b, 3, bdims, bstr, bbox))
      KSB_FAIL(KS_ERROR_INTERNAL, std::string(a.where) + ": tensor map for B rejected");
  } else {
  {
    const uint64_t dims[2] = {static_cast<uint64_t>(a.k), static_cast<uint64_t>(a.m)};
    const uint64_t str[1] = {static_cast<uint64_t>(a.k)};
    const uint32_t box[2] = {static_cast<uint32_t>(kBK), static_cast<uint32_t>(kBM)};
    const uint32_t box32[2] = {static_cast<uint32_t>(kBK), 32u};
    if (!encode_u8(&tm_a, a.a, 2, dims, str, box) || !encode_u8(&tm_a32, a.a, 2, dims, str, box32))
      KSB_FAIL(KS_ERROR_INTERNAL, std::string(a.where) + ": tensor map for A rejected");
  }
  if (a.nt) {
    const uint64_t dims[3] = {static_cast<uint64_t>(a.k), static_cast<uint64_t>(a.n), static_cast<uint64_t>(experts)};
    const uint64_t str[2] = {static_cast<uint64_t>(a.k), static_cast<uint64_t>(a.k) * static_cast<uint64_t>(a.n)};
    const uint32_t box[3] = {static_cast<uint32_t>(kBK), static_cast<uint32_t>(bn), 1u};
    if (!encode_u8(&tm_b, a.b, 3, dims, str, box))
      KSB_FAIL(KS_ERROR_INTERNAL, std::string(a.where) + ": tensor map for B rejected");
  } else {
    const uint64_t dims[3] = {static_cast<uint64_t>(a.n), static_cast<uint64_t>(a.k), static_cast<uint64_t>(experts)};
    const uint64_t str[2] = {static_cast<uint64_t>(a.n), static_cast<uint64_t>(a.k) * static_cast<uint64_t>(a.n)};
    const uint32_t box[3] = {128u, static_cast<uint32_t>(kBK), 1u};
    if (!encode_u8(&tm_b, a.b, 3, dims, str, box))
      KSB_FAIL(KS_ERROR_INTERNAL, std::string(a.where) + ": tensor map for B rejected");
  }
  }

  Params p;
  p.out = a.out;
  p.a_scale = a.a_scale;
  p.b_scale = a.b_scale;
  p.offsets = a.offsets;
  p.as_row_stride = a.a_scale_ld > 0 ? 1 : (a.k + kBK - 1) / kBK;
  p.as_kb_stride = a.a_scale_ld > 0 ? a.a_scale_ld : 1;
  p.masked_m = a.masked_m;
  p.max_m = static_cast<int>(a.max_m);
  p.bias = a.bias;
  p.rows_per_part = a.num_out_parts > 0 ? static_cast<int>(a.rows_per_part) : 0;
  for (int i = 0; i < kMaxOutParts; ++i) p.out_parts[i] = i < a.num_out_parts ? a.out_parts[i] : nullptr;
  p.a_per_row = a.a_per_row ? 1 : 0;
  p.b_per_col = a.b_per_col ? 1 : 0;
  p.fault_word = kernel_fault_word();
  p.num_experts = experts;
  p.m = static_cast<int>(a.m);
  p.n = static_cast<int>(a.n);
  p.k = static_cast<int>(a.k);
  p.nkb = static_cast<int>((k_bytes + kBK - 1) / kBK);
  p.nnb = static_cast<int>((a.n + 127) / 128);
  p.tiles_n = static_cast<int>((a.n + bn - 1) / bn);
  p.tiles_m = static_cast<int>((a.m + kBM - 1) / kBM);
  // operand formats: e4m3 / e5m2 for the fp8 kinds; signed 8-bit integers with an int32
  // accumulator for kind::i8
  // (kind::f16: 0 = f16, 1 = bf16)
  const uint32_t fmt = a.mode == 2 ? 1u : (a.mode == 3 ? (a.out_dtype == KS_DTYPE_BF16 ? 1u : 0u) : (a.e5m2 ? 1u : 0u));
  p.idesc = umma_instr_desc(fmt, fmt, 0u, a.nt ? 0u : 1u, kBM, static_cast<uint32_t>(bn), a.mode == 2 ? 2u : 1u);
  const size_t out_elt = a.out_dtype == KS_DTYPE_F32 ? 4 : 2;
  bool out_aligned = a.num_out_parts > 0 ? true : aligned16(a.out);
  for (int i = 0; i < a.num_out_parts; ++i) out_aligned = out_aligned && aligned16(a.out_parts[i]);
  p.vec_store = (out_aligned && (static_cast<size_t>(a.n) * out_elt) % 16 == 0) ? 1 : 0;

  int64_t tiles = tiles_m_bound * p.tiles_n;
  const int grid = static_cast<int>(cluster_s > 1 ? tiles * cluster_s : (tiles < sms ? (tiles < 1 ? 1 : tiles) : sms));

  // K-split of the last partial round (dense problems only). Worth it when the tiles left
  // over after the full rounds occupy at most half of the CTAs and every part keeps at least
  // four K-blocks; the part count is capped at eight (each part is one more partial to read).
  p.split_from = static_cast<int>(tiles);
  p.split_items = 0;
  p.split_s = 1;
  p.split_slots = nullptr;
  std::optional<StreamScratch> scratch;
  p.cluster_s = cluster_s;
  if (cluster_s > 1) {
    p.split_from = 0;
    p.split_items = grid;
    p.split_s = cluster_s;
  } else if (!grouped && a.mode == 0 && a.force_split != 0 && a.num_out_parts == 0 && tiles > grid) {
    const int rem = static_cast<int>(tiles % grid);
    const int s = rem > 0 ? split_parts(grid, rem, p.nkb) : 1;
    if (rem > 0 && s >= 2) {
      const size_t slot_bytes = static_cast<size_t>(rem) * s * kBM * bn * sizeof(float);
      scratch.emplace(stream);   // (until both kernels are enqueued)
      float4* slots = static_cast<float4*>(scratch->get(slot_bytes, 2));
      if (slots != nullptr) {
        p.split_from = static_cast<int>(tiles) - rem;
        p.split_items = rem * s;
        p.split_s = s;
        p.split_slots = slots;
      }
    }
  }
  return bn == 256 ? launch_bn<256>(a, tm_a, tm_a32, tm_b, p, grid, stream) : launch_bn<128>(a, tm_a, tm_a32, tm_b, p, grid, stream);
}

}  // namespace sm100
}  // namespace ksb
