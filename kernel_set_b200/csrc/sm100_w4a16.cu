// int4 weight-only GEMM for sm_100a: any number of rows, scale groups of 32, 64 or a multiple
// of 128.
//
// Computes what ks_gemm_w4a16 declares (reference: kernels/src/gemm/
// gemm_w4a16.cu:50-130, layout :6-19): C[M,N] = A[M,K] . W + bias with
// W[k,n] = (q[k,n] - zero[g,n]) * scale[g,n] rounded once to the activation
// type (the reference's torch statement, benchmarks/bench.py:1275-1284), then
// multiplied with fp32 accumulation.
//
// The GEMM is transposed onto the tensor core: the weight's N dimension is the
// UMMA M dimension (128 TMEM lanes), the tokens are the UMMA N dimension
// (16..192 columns), so a CTA streams 128 weight columns x 128 k per step ("unit").
//   warp 0        weight producer (TMA): boxes of two K-steps, [128 byte-rows x 128
//                 columns] = 16 KB straight from HBM. (A warp keeps only
//                 about three TMA loads in flight whatever their size; 8 KB boxes cap a
//                 single producer warp near 2.5 TB/s, 16 KB boxes near 4.5 TB/s.)
//   warp 2        activation producer (TMA): [tokens x 64 or 128 k] from L2
//   warps 4-19    dequantisation (see there): shared memory -> tensor memory, where the MMA
//                 reads the weights as its A operand
//   warps 1, 3    MMA issuers on alternate units (above 128 tokens: on the two 64-k halves of every unit)
//   the rest      epilogue: tensor memory -> registers -> C, or an fp32 partial
// Work is dealt out in one of three ways, chosen by estimated time (geometry_of): a tile's
// K range over a cluster of CTAs that add their partial sums over distributed shared memory; equal
// contiguous runs of units per CTA, where a tile shared by several CTAs is finished by the last to
// arrive (fp32 slots in stream scratch, added in slot order: deterministic); runs of whole tiles.
//
// What bounds it, from work-skipping builds at K=8192, N=18944 (one tile of 64 units per CTA, 82 MB:
// 12.6 us at the HBM rate). 16 tokens: 42 us, without the dequantisation arithmetic 26, without the
// arithmetic and seven of eight MMAs 22: the integer pipe (half rate) and instruction issue of
// sixteen warps. Wide tiles: the stream from L2 (8 KB of weight and 256 bytes per token a unit), the MMAs (4
// cycles per token and unit) and the arithmetic overlap only partly.
// Measured, 128-row tiles with the weights through shared memory -> this design: K=4096 N=28672
// M=2048 545 -> 416 us (1.16 PFLOP/s), M=192 92 -> 49 us; M=100 N=11008 group 64 730 -> 22.5 us
// (narrow groups ran on the SIMT kernel); K=N=4096 M=1 12.3 -> 9.4 us.
//
// Roofline: HBM-bound for M <= 64; algorithmic bytes per launch
// K*N/2 + (K/gs)*N*2*(1 or 2) + M*K*2 + M*N*2.
#include <cstdio>
#include <mutex>

#include <cstdlib>

#include "common.cuh"
#include "sm100_host.cuh"
#include "sm100_ptx.cuh"
#include "sm100_w4a16.cuh"

namespace ksb {
namespace sm100 {
namespace {

constexpr int kTileN = 128;    // weight columns per tile = UMMA M
constexpr int kStepK = 128;    // k per pipeline step ("unit" = 128 columns x 128 k)
constexpr int kRawBytes = (kStepK / 2) * kTileN;      // 8192
constexpr int kRawStageBytes = 2 * kRawBytes;         // one TMA box: two K-steps
constexpr int kDeqWarps = 16;      // dequantising warps, in two or four groups (see Cfg)
constexpr int kDeqStages = 4;      // operand stages in tensor memory
constexpr int kAtomK = 64;         // k per 128-byte swizzle atom of the activations

// Everything that depends on the width of the token tile. The numbers of operand stages and
// of activation stages must be multiples of the number of issuers: an issuer's wait on a
// stage's `full` barrier is ordered after the stage's previous use only because the same
// issuer consumed that use. (Three issuers with four stages let an issuer pass a fresh barrier
// one phase early: intermittent bounded-wait timeouts on the GPU, and a deadlock in the
// protocol model under tests/.)
template <int MTMAX, bool FINE>
struct Cfg {
  // Dequantisation: a warp takes one TMEM lane quarter (32 columns) of its group's unit. Above 32
  // tokens two groups of eight warps take alternate units, a warp one 64-k half: with four
  // operand stages a group has two of its own and fills one while the MMAs read the other. (Four groups of
  // four are each tied to one stage: a group's next unit waits for the MMAs of its last, and the
  // two times add up.) Up to 32 tokens the MMAs are short, and what counts is the work per warp and
  // unit outside the cells (waits, scales, their tests: ~100 of 230 instructions): four groups, a warp
  // takes both halves. K=14336 N=28672 M=24: 92.9 us with two groups, 78.7 with four; K=14336 N=4096 M=1 19.8
  // and 17.6. Scale groups of 32 and 64 (FINE) need two constants per half, gain 1-2 % or lose it, and stay.
  static constexpr int kGroups = MTMAX <= 32 && !FINE ? 4 : 2;
  static constexpr int kDeqGroupWarps = kDeqWarps / kGroups;
  static constexpr int kKHalves = kGroups / 2;   // 64-k halves of a unit that a warp takes
  // Issuing a tcgen05.mma costs its thread ~55 cycles: up to 64 token columns the tensor core needs
  // less than that, at 128 about as much. Two issuers, with accumulators of their own, take alternate
  // units, or above 128 rows the two 64-k halves of every unit (kHalfStages): the operand ring's 128
  // columns are then four stages of 64 k, each filled by four warps. (One issuer for both halves: K=4096
  // N=28672 M=2048 445 us instead of 416.)
  // Two sums also halve the error. tcgen05.mma truncates what it adds up, so a sum's error grows with its
  // instructions: at K=14336, f16, positive operands, 256-row tiles, which leave room for one accumulator, had
  // 10.2 % of the results an ulp off, the tile of 192 rows 5.4 %. (256 rows take 370 us. Parking the sums
  // of the first half of K in L2, 128 KB a tile, made that 460.)
  static constexpr int kIssuers = 2;
  static constexpr bool kHalfStages = MTMAX > 128;
  // Consecutive instructions into one accumulator wait for one another; with 32 columns that
  // latency would set the pace, so an issuer alternates between two.
  static constexpr int kAccsPerIssuer = MTMAX <= 32 ? 2 : 1;
  static constexpr int kAccs = kIssuers * kAccsPerIssuer;
  // Tensor memory: 256 columns of operand ring, 256 of accumulators: two segment buffers up to
  // 64 token columns, one above (the epilogue of a tile, ~2 % of a K = 4096 tile, is then
  // not overlapped with the next tile's MMAs).
  static constexpr int kAccBufs = MTMAX <= 64 ? 2 : 1;
  static constexpr int kAccCols = kAccBufs * kAccs * MTMAX;
  static constexpr int kOperandCol0 = kAccCols;
  static constexpr int kDeqPerUnit = kHalfStages ? 2 : 1;            // operand stages per unit
  static constexpr int kDeqTmemCols = kStepK / 2 / kDeqPerUnit;      // of two k each
  static constexpr int kTmemCols = 512;
  static_assert(kAccCols + kDeqStages * kDeqTmemCols <= 512, "TMEM holds 512 columns");
  // Activations: a stage is a whole unit (both 64-k atoms), or one atom with half stages, which the
  // commit that frees the operand stage frees too.
  static constexpr int kActAtoms = kHalfStages ? 1 : 2;       // atoms per stage
  static constexpr int kActPerUnit = 2 / kActAtoms;           // stages per unit
  static constexpr int kActStage = MTMAX * kAtomK * 2 * kActAtoms;
  static constexpr int kActStages = MTMAX <= 32 ? 8 : (MTMAX <= 64 ? 6 : 4);
  static constexpr int kRawStages = MTMAX <= 32 ? 8 : (MTMAX <= 64 ? 7 : 5);
  static_assert(kDeqStages % kIssuers == 0 && kActStages % kIssuers == 0, "see above");
  static_assert(!kHalfStages || kActStages == kDeqStages, "one barrier frees a stage of either");
  static constexpr int kEpiWarps = MTMAX <= 128 ? 4 : 8;      // 192 tokens: two warps share a lane quarter
  static constexpr int kEpiThreads = kEpiWarps * 32;
  static constexpr int kThreads = 128 + kDeqWarps * 32 + kEpiThreads;
  static constexpr int kRing = kActStages * kActStage + kRawStages * kRawStageBytes;
  static constexpr int kNumBars = 2 * kRawStages + 2 * kActStages + 2 * kDeqStages + 2 * kAccBufs;
  static constexpr int kSmemBytes = kRing + 1024 + 512;
  static_assert(8 * kNumBars + 16 <= 512 && kSmemBytes <= 232448, "shared memory layout");
};

struct Params {
  void* c;
  const void* bias;
  const void* scales;
  const void* zeros;
  float* slots;             // fp32 partials, [slot][mt / 4][128][4]
  unsigned int* counters;
  unsigned int* fault_word;
  int m, n, k;
  int mt;                   // token tile, multiple of 16, <= MTMAX
  int m_tiles;
  int n_tiles;
  int k_steps;              // 128-k steps, rounded up to an even number (a box holds two)
  int gs_steps;             // K-steps per scale group (group_size / 128); FINE: unused
  int sub_shift;            // FINE: log2 of the 32-k quarters per scale group (group_size 32: 0, 64: 1)
  int groups;               // rows of scales and zeros
  int split;                // 1: equal runs of units, tiles may be shared by CTAs; 0: whole tiles
  int cluster_s;            // > 1: every tile is one cluster's, its K range cut over the cluster's CTAs
  int c_vec;                // C is 8-byte aligned
  int has_zeros;
  uint32_t idesc;
};

template <typename T> struct Pack16;
template <> struct Pack16<__nv_bfloat16> {
  using V2 = __nv_bfloat162;
  static constexpr float kMaxZero = 127.0f;             // zero-points up to here: |q - zero| is exact
  static constexpr float kUnit = 0x1p-133f;             // the bit pattern q is q * 2^-133 (subnormal)
  static constexpr float kUp = 0x1p127f;                // largest power of two; q * kUnit * kUp = q / kDown
  static constexpr float kDown = 0x1p6f;
  __device__ static V2 from_bits(uint32_t b) { return *reinterpret_cast<V2*>(&b); }
  __device__ static uint32_t bits(V2 v) { return *reinterpret_cast<uint32_t*>(&v); }
  __device__ static V2 splat(float f) { return __float2bfloat162_rn(f); }
  __device__ static float lo(V2 v) { return __low2float(v); }
  __device__ static float hi(V2 v) { return __high2float(v); }
  __device__ static V2 make(float a, float b) { return __floats2bfloat162_rn(a, b); }
  __device__ static V2 low(V2 v) { return __low2bfloat162(v); }    // the low half twice
  __device__ static V2 high(V2 v) { return __high2bfloat162(v); }
};
template <> struct Pack16<__half> {
  using V2 = __half2;
  static constexpr float kMaxZero = 1023.0f;
  static constexpr float kUnit = 0x1p-24f;
  static constexpr float kUp = 0x1p15f;
  static constexpr float kDown = 0x1p9f;
  __device__ static V2 from_bits(uint32_t b) { return *reinterpret_cast<V2*>(&b); }
  __device__ static uint32_t bits(V2 v) { return *reinterpret_cast<uint32_t*>(&v); }
  __device__ static V2 splat(float f) { return __float2half2_rn(f); }
  __device__ static float lo(V2 v) { return __low2float(v); }
  __device__ static float hi(V2 v) { return __high2float(v); }
  __device__ static V2 make(float a, float b) { return __floats2half2_rn(a, b); }
  __device__ static V2 low(V2 v) { return __low2half2(v); }
  __device__ static V2 high(V2 v) { return __high2half2(v); }
};

// prmt with all four selector bits (bit 3 of a nibble replicates the byte's sign bit).
__device__ __forceinline__ uint32_t byte_perm_sign(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Weight column (inside a warp's 32) that TMEM lane `lane` of the warp's quarter holds: the
// store shape of the dequantised operand puts columns 2g and 2g + 1 of a block of 16 in lanes
// g and g + 8 (see the dequantisation role).
__device__ __forceinline__ int column_of_lane(int lane) { return (lane & 16) + 2 * (lane & 7) + ((lane >> 3) & 1); }

// Stores 16 token rows x the warp's 32 columns: a lane holds its column of token j in v[j].
// Two exchanges with the lanes of the neighbouring columns turn that into four adjacent columns
// of four tokens per lane, so that a store instruction writes 64 contiguous bytes of four rows
// instead of 64 bytes of one. `c` points at (first token, first column of the warp).
template <typename T>
__device__ __forceinline__ void store_tokens16(T* c, int ld, const float (&v)[16], int lane, int rows_ok, int cols_ok,
                                               bool vec) {
  if (!vec) {
    const int col = column_of_lane(lane);
    if (col < cols_ok) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < rows_ok) c[static_cast<size_t>(j) * ld + col] = from_f32<T>(v[j]);
    }
    return;
  }
  using P = Pack16<T>;
  // w[i] = tokens (2i, 2i + 1) of this lane's column
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = P::bits(P::make(v[2 * i], v[2 * i + 1]));
  // columns 2g and 2g + 1 (lanes g, g + 8): the first lane keeps token 2i of both, the other token 2i + 1
  const bool odd = (lane & 8) != 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, w[i], 8);
    w[i] = odd ? __byte_perm(other, w[i], 0x7632) : __byte_perm(w[i], other, 0x5410);
  }
  // column pairs g and g + 1: even lanes keep the pairs i < 4, odd lanes i >= 4
  const bool up = (lane & 1) != 0;
  const int col = (lane & 16) + 2 * (lane & 6);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t give = up ? w[i] : w[i + 4];
    const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 1);
    const uint32_t keep = up ? w[i + 4] : w[i];
    const int token = 2 * (i + (up ? 4 : 0)) + (odd ? 1 : 0);
    if (token < rows_ok && col < cols_ok)
      *reinterpret_cast<uint2*>(c + static_cast<size_t>(token) * ld + col) =
          up ? make_uint2(got, keep) : make_uint2(keep, got);
  }
}

// FINE: scale groups of 32 or 64 k (several per K-step); otherwise multiples of 128.
template <typename T, int MTMAX, bool FINE>
__global__ void __launch_bounds__((Cfg<MTMAX, FINE>::kThreads), 1)
w4a16_umma_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a,
                  const Params p) {
  using C = Cfg<MTMAX, FINE>;
  using P16 = Pack16<T>;
  using V2 = typename P16::V2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw_addr);
  // ring: activation stages | raw stages | barriers
  const uint32_t act_base = base;
  const uint32_t rawst_base = act_base + C::kActStages * C::kActStage;
  const uint32_t bar_base = rawst_base + C::kRawStages * kRawStageBytes;
  uint8_t* ctrl_ptr = base_ptr + (bar_base - base);
  const uint32_t bar_raw_full = bar_base;
  const uint32_t bar_raw_empty = bar_raw_full + 8 * C::kRawStages;
  const uint32_t bar_act_full = bar_raw_empty + 8 * C::kRawStages;
  const uint32_t bar_act_empty = bar_act_full + 8 * C::kActStages;
  const uint32_t bar_deq_full = bar_act_empty + 8 * C::kActStages;
  const uint32_t bar_deq_empty = bar_deq_full + 8 * kDeqStages;
  const uint32_t bar_acc_full = bar_deq_empty + 8 * kDeqStages;
  const uint32_t bar_acc_empty = bar_acc_full + 8 * C::kAccBufs;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ctrl_ptr + 8 * C::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* last_flag = tmem_slot + 2;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitCtx wctx{smem_u32(const_cast<uint32_t*>(abort_flag)), p.fault_word};

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kRawStages; ++s) {
      mbar_init(bar_raw_full + 8 * s, 1);
      mbar_init(bar_raw_empty + 8 * s, 2 * C::kDeqGroupWarps);   // both halves of a box
    }
    for (int s = 0; s < C::kActStages; ++s) {
      mbar_init(bar_act_full + 8 * s, 1);
      mbar_init(bar_act_empty + 8 * s, 1);   // the issuer that owns the unit (half stages: not used)
    }
    for (int s = 0; s < kDeqStages; ++s) {
      mbar_init(bar_deq_full + 8 * s, C::kDeqGroupWarps / C::kDeqPerUnit);
      mbar_init(bar_deq_empty + 8 * s, 1);
    }
    for (int b = 0; b < C::kAccBufs; ++b) {
      mbar_init(bar_acc_full + 8 * b, C::kIssuers);
      mbar_init(bar_acc_empty + 8 * b, C::kEpiWarps);
    }
    *abort_flag = 0u;
    fence_barrier_init();
    prefetch_tensormap(&tm_w);
    prefetch_tensormap(&tm_a);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // Unit space: (column tile, token tile, K-step), K-step fastest; a "tile" below is a
  // (column tile, token tile) pair. Token tiles of one column tile are neighbours, so the
  // CTAs in flight share weights. Units are dealt in equal contiguous runs (tiles may be
  // split between CTAs), or in runs of whole tiles (split == 0), or, where there are few
  // tiles, a tile's units over the CTAs of a cluster.
  const long long tiles = static_cast<long long>(p.n_tiles) * p.m_tiles;
  const long long units = tiles * p.k_steps;
  const int ctas = gridDim.x;
  long long u_begin, u_end;
  if (p.cluster_s > 1) {
    // (parts are whole boxes of two steps)
    const int part = static_cast<int>(blockIdx.x) % p.cluster_s;
    const long long tile_begin = static_cast<long long>(blockIdx.x) / p.cluster_s * p.k_steps;
    u_begin = tile_begin + 2 * (part * (p.k_steps / 2) / p.cluster_s);
    u_end = tile_begin + 2 * ((part + 1) * (p.k_steps / 2) / p.cluster_s);
  } else if (p.split) {
    u_begin = run_start(units, ctas, blockIdx.x);
    u_end = run_start(units, ctas, blockIdx.x + 1);
  } else {
    u_begin = run_start(tiles, ctas, blockIdx.x) * p.k_steps;
    u_end = run_start(tiles, ctas, blockIdx.x + 1) * p.k_steps;
  }
  // The next kernel on the stream may start its prologue now. This one touches what the
  // kernel before it may have produced or may still read (activations, C, the split-K
  // scratch) only behind grid_dependency_wait(): the activation producer and the epilogue.
  grid_launch_dependents();

  if (warp == 0) {
    // ------------------------- weight producer (TMA) -------------------------
    // boxes of two K-steps; k_steps is even, so a box never straddles two tiles
    const long long b_end = (u_end + 1) >> 1;
    uint32_t itb = 0;
    // (tile, step) advance with the loop: a 64-bit division per box would cost hundreds of cycles
    const long long t0 = (u_begin & ~1ll) / p.k_steps;
    int step = static_cast<int>((u_begin & ~1ll) - t0 * p.k_steps);
    int ntile = static_cast<int>(t0 / p.m_tiles);
    int mtile = static_cast<int>(t0 - static_cast<long long>(ntile) * p.m_tiles);
    for (long long b = u_begin >> 1; b < b_end; ++b, ++itb, step += 2) {
      if (step >= p.k_steps) {
        step -= p.k_steps;
        if (++mtile == p.m_tiles) { mtile = 0; ++ntile; }
      }
      const uint32_t sr = itb % C::kRawStages, pr = (itb / C::kRawStages) & 1u;
      if (!mbar_wait(wctx, bar_raw_empty + 8 * sr, pr ^ 1u, 0x100u + sr)) break;
      const uint32_t full = bar_raw_full + 8 * sr;
      mbar_arrive_expect_tx_elect(full, 2 * kRawBytes);
      tma_load_2d_elect(rawst_base + sr * kRawStageBytes, &tm_w, full, ntile * kTileN, step * (kStepK / 2));
    }
  } else if (warp == 2) {
    // ----------------------- activation producer (TMA) -----------------------
    grid_dependency_wait();
    const uint32_t act_tx = static_cast<uint32_t>(p.mt) * kAtomK * 2 * C::kActAtoms;
    const long long t0 = u_begin / p.k_steps;
    int step = static_cast<int>(u_begin - t0 * p.k_steps);
    int mtile = static_cast<int>(t0 % p.m_tiles);
    uint32_t ita = 0;
    bool ok = true;
    for (long long u = u_begin; ok && u < u_end; ++u) {
#pragma unroll
      for (int h = 0; h < C::kActPerUnit; ++h, ++ita) {
        const uint32_t sa = ita % C::kActStages, pa = (ita / C::kActStages) & 1u;
        if (!mbar_wait(wctx, (C::kHalfStages ? bar_deq_empty : bar_act_empty) + 8 * sa, pa ^ 1u, 0x180u + sa)) {
          ok = false;
          break;
        }
        const uint32_t full = bar_act_full + 8 * sa;
        mbar_arrive_expect_tx_elect(full, act_tx);
        // the map views A as [K/64][M][64]
        tma_load_3d_elect(act_base + sa * C::kActStage, &tm_a, full, 0, mtile * p.mt, step * 2 + h);
      }
      if (++step == p.k_steps) {
        step = 0;
        if (++mtile == p.m_tiles) mtile = 0;
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------ MMA issuers ------------------------------
    // The issuers take the units in turn (unit it -> issuer it % kIssuers; half stages: the halves): per unit an
    // issuer pays its barrier tests (~100 cycles each), eight MMAs and the commits; sharing
    // every unit between all issuers made each of them pay the fixed part for every unit. An
    // issuer owns its accumulator(s) of the segment buffer and tells the epilogue "done" after
    // its last unit of the segment; an issuer without a unit in a short segment arrives
    // without a commit, and the epilogue skips its accumulators.
    const int me = warp == 1 ? 0 : 1;
    uint32_t it = 0, seg = 0;
    int step = static_cast<int>(u_begin % p.k_steps);
    uint32_t n_in_seg = 0;
    for (long long u = u_begin; u < u_end; ++u, ++it, step = (step + 1 == p.k_steps) ? 0 : step + 1) {
      const bool seg_first = (u == u_begin) || (step == 0);
      const bool seg_last = (u + 1 == u_end) || (step == p.k_steps - 1);
      // last unit of this segment: end of the tile or of this CTA's run
      const long long tile_last = u - step + p.k_steps - 1;
      const long long seg_last_u = tile_last < u_end - 1 ? tile_last : u_end - 1;
      const bool mine = C::kHalfStages || static_cast<int>(it % C::kIssuers) == me;
      const bool my_last = u + (C::kHalfStages ? 1 : C::kIssuers) > seg_last_u;   // no later unit of mine in this segment
      const uint32_t buf = seg % C::kAccBufs, pacc = (seg / C::kAccBufs) & 1u;
      if (seg_first) n_in_seg = 0;
      if (mine) {
        if (n_in_seg == 0 && !mbar_wait(wctx, bar_acc_empty + 8 * buf, pacc ^ 1u, 0x200u + buf)) break;
        const uint32_t d_tmem = tmem_base + buf * (C::kAccs * MTMAX);
        const uint32_t its = C::kHalfStages ? it * 2 + me : it;   // stage in order of use
        const uint32_t sd = its % kDeqStages, pd = (its / kDeqStages) & 1u;
        const uint32_t sa = its % C::kActStages, pa = (its / C::kActStages) & 1u;
        if (!mbar_wait_both(wctx, bar_deq_full + 8 * sd, pd, 0x280u + sd, bar_act_full + 8 * sa, pa, 0x300u + sa)) break;
        tc_fence_after_sync();
        const uint32_t a_src = act_base + sa * C::kActStage;
        const uint32_t w_stage = tmem_base + C::kOperandCol0 + sd * C::kDeqTmemCols;
#pragma unroll
        for (int kk = 0; kk < 4 * C::kActAtoms; ++kk) {
          // tokens: K-major, 64-k atoms of mt rows, 32 B per instruction inside an atom;
          // weights: 16 k = 8 columns of the operand stage in tensor memory
          const uint64_t a_desc = umma_smem_desc_sw128(a_src + (kk >> 2) * (p.mt * 128) + (kk & 3) * 32, 16, 1024);
          const uint32_t d_acc = d_tmem + (me * C::kAccsPerIssuer + (kk % C::kAccsPerIssuer)) * MTMAX;
          umma_f16_tmem_a_elect(d_acc, w_stage + kk * 8, a_desc, p.idesc,
                                (n_in_seg == 0 && kk < C::kAccsPerIssuer) ? 0u : 1u);
        }
        tc_commit_elect(bar_deq_empty + 8 * sd);
        if constexpr (!C::kHalfStages) tc_commit_elect(bar_act_empty + 8 * sa);
        ++n_in_seg;
        if (my_last) tc_commit_elect(bar_acc_full + 8 * buf);   // my last unit of the segment
      } else if (seg_last && n_in_seg == 0) {
        // A short segment without a unit of mine. Like an issuer with work, wait until the
        // epilogue has drained this buffer's previous segment: otherwise this arrival could
        // overtake my own (asynchronous) commit for that segment and complete its phase early.
        if (!mbar_wait(wctx, bar_acc_empty + 8 * buf, pacc ^ 1u, 0x200u + buf)) break;
        mbar_arrive_elect(bar_acc_full + 8 * buf);
      }
      if (seg_last) ++seg;
    }
  } else if (warp >= 4 && warp < 4 + kDeqWarps) {
    // ----------------------------- dequantisation -----------------------------
    // A packed byte holds the codes of k and k+1 of one column, which is exactly one 32-bit
    // operand cell. ldmatrix.trans hands lane (g = lane / 4, s = lane % 4) a word with the bytes
    // (row 2s, columns 2g, 2g + 1) and (row 2s + 1, columns 2g, 2g + 1) of an 8-row x 16-column
    // block; tcgen05.st.16x256b takes from it the cells (TMEM lane g, columns 2s, 2s + 1) and
    // (lane g + 8, columns 2s, 2s + 1). So TMEM lanes g and g + 8 stand for the weight columns 2g
    // and 2g + 1, and no byte crosses a lane. The low and the high nibbles of the word are split once;
    // per cell one byte permute then puts code k into the low half and code k+1 into the high
    // half. Such a half, read as a 16-bit float, is the subnormal q * kUnit, and one exact
    // multiply-add makes it (q - zero) / kDown; the product with kDown * scale rounds once, as
    // (q - zero) * scale does. (Building the float magic + q first costs one more integer
    // instruction per cell, and the integer pipe is what bounds this loop.)
    // (Reading one byte per lane and row instead takes a full shared-memory cycle for 32 bytes,
    // 256 per unit, on the port through which the MMAs read 64 KB and TMA writes 72 KB per unit.)
    // The loop is bound by instruction issue (the integer pipe at half rate above all), so
    // everything outside the cells counts: 32-bit counters relative to the CTA's run, ring
    // positions that advance instead of divisions, addresses of the scale rows that advance, and
    // zero-points tested two columns at a time.
    constexpr int kGroups = C::kGroups, kBoxStep = kGroups / 2;
    const int group = (warp - 4) / C::kDeqGroupWarps;
    const int half = group & 1;                 // K-step half of the group's boxes = parity of its units
    const int box0 = group >> 1;                // first box: of four groups, two take every other box
    const int khalf = C::kKHalves == 2 ? 0 : ((warp - 4) >> 2) & 1;   // (first) 64-k half of the unit
    static_assert(P16::kUnit * P16::kUp * P16::kDown == 1.0f, "the three factors cancel");
    const V2 up2 = P16::splat(P16::kUp), down2 = P16::splat(P16::kDown), neg_inv_down2 = P16::splat(-1.0f / P16::kDown);
    const V2 max_zero2 = P16::splat(P16::kMaxZero), zero2 = P16::from_bits(0u);
    const V2 max_scale2 = P16::splat(P16::kUp);
    const V2 whole2 = P16::splat(P16::kMaxZero + 1.0f);   // adding it rounds to whole numbers
    const int quarter = warp & 3;
    constexpr int kSz = FINE ? 2 : 1;           // scale rows of this warp's k: one per 32 k (FINE: 64 k), or one
    static_assert(!FINE || C::kKHalves == 1, "see above");
    const int col0 = quarter * 32 + 2 * (lane >> 2);   // this lane's columns: col0, col0 + 1, col0 + 16, col0 + 17
    const int n_units = static_cast<int>(u_end - u_begin);
    const int odd0 = static_cast<int>(u_begin & 1);
    const int n_boxes = (n_units + odd0 + 1) >> 1;
    // Scales and zero-points come straight from global memory, fetched one unit of the group
    // ahead (k_steps and kGroups are even, so the parity of step is fixed).
    int it = 2 * box0 + half - odd0;            // unit of the first box, relative to the run; -1: a neighbour's
    const long long u_first = u_begin + (it < 0 ? it + kGroups : it);
    const long long f_t0 = u_first / p.k_steps;
    int f_step = static_cast<int>(u_first - f_t0 * p.k_steps);
    int f_ntile = static_cast<int>(f_t0 / p.m_tiles);
    int f_mtile = static_cast<int>(f_t0 - static_cast<long long>(f_ntile) * p.m_tiles);
    int f_row = FINE ? 0 : f_step / p.gs_steps, f_in_row = FINE ? 0 : f_step - f_row * p.gs_steps;
    uint32_t s_pair[kSz][2], z_pair[kSz][2];   // [scale row][block of 16 columns]: columns 2g (low half), 2g + 1
#pragma unroll
    for (int i = 0; i < kSz; ++i) s_pair[i][0] = s_pair[i][1] = z_pair[i][0] = z_pair[i][1] = 0u;
    auto fetch = [&]() {
      const int n = f_ntile * kTileN + col0;
#pragma unroll
      for (int i = 0; i < kSz; ++i) {
        const int row = FINE ? ((f_step * 4 + khalf * 2 + i) >> p.sub_shift) : f_row;
        const long long idx = static_cast<long long>(row) * p.n + n;
        const unsigned short* gs = static_cast<const unsigned short*>(p.scales) + idx;
        const unsigned short* gz = static_cast<const unsigned short*>(p.zeros) + idx;
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          // (the step that rounds k_steps up to an even number has no row: codes and activations
          // are zero-filled there, and zero scales keep the product zero)
          const bool in = n + 16 * cb < p.n && row < p.groups;
          s_pair[i][cb] = in ? __ldg(reinterpret_cast<const unsigned int*>(gs + 16 * cb)) : 0u;
          if (p.has_zeros) z_pair[i][cb] = in ? __ldg(reinterpret_cast<const unsigned int*>(gz + 16 * cb)) : 0u;
        }
      }
    };
    auto fetch_advance = [&]() {
      f_step += kGroups;
      if (f_step >= p.k_steps) {
        do {   // (a tile may have fewer K-steps than there are groups)
          f_step -= p.k_steps;
          if (++f_mtile == p.m_tiles) { f_mtile = 0; ++f_ntile; }
        } while (f_step >= p.k_steps);
        if constexpr (!FINE) {
          f_row = 0;
          f_in_row = f_step;
        }
      } else if constexpr (!FINE) {
        f_in_row += kGroups;
      }
      if constexpr (!FINE) {
        while (f_in_row >= p.gs_steps) { f_in_row -= p.gs_steps; ++f_row; }
      }
    };
    if (u_first < u_end) fetch();
    // ldmatrix row addresses: lanes 0-7 / 8-15 rows 0-7 of the first / second block of 16
    // columns, lanes 16-31 the same of rows 8-15; 128-byte rows with the 16-byte chunks swizzled
    const uint32_t lane_off =
        static_cast<uint32_t>(half * kRawBytes + khalf * (32 * 128) + ((lane >> 4) * 8 + (lane & 7)) * 128 +
                              (((quarter * 2 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
    const uint32_t lane_dst = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::kOperandCol0 +
                              (C::kHalfStages ? 0 : khalf * 32);
    static_assert(C::kRawStages % kBoxStep == 0, "a group keeps to its raw stages");
    uint32_t stage = box0, phase = 0;
    for (int b = box0; b < n_boxes; b += kBoxStep, it += kGroups) {
      const uint32_t sr = stage, pr = phase;
      stage += kBoxStep;
      if (stage >= C::kRawStages) { stage -= C::kRawStages; phase ^= 1u; }
      if (it < 0 || it >= n_units) {
        // this half of the box belongs to a neighbouring CTA's run
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_raw_empty + 8 * sr);
        continue;
      }
      const uint32_t its = C::kHalfStages ? it * 2 + khalf : it;
      const uint32_t sd = its & (kDeqStages - 1), pd = (its / kDeqStages) & 1u;
      static_assert((kDeqStages & (kDeqStages - 1)) == 0, "a power of two");
      // constants of the unit: columns 2g, 2g + 1 of the first block of 16, then of the second
      V2 sd2[kSz][2], zd2[kSz][2];     // scale * kDown, -zero / kDown
      uint32_t s_cur[kSz][2], z_cur[kSz][2];
      bool simple_lane = true;
#pragma unroll
      for (int i = 0; i < kSz; ++i) {
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          s_cur[i][cb] = s_pair[i][cb];
          z_cur[i][cb] = z_pair[i][cb];
          const V2 sv = P16::from_bits(s_cur[i][cb]), zv = P16::from_bits(z_cur[i][cb]);
          sd2[i][cb] = __hmul2(sv, down2);
          zd2[i][cb] = __hmul2(zv, neg_inv_down2);
          // exact for integer zero-points 0..kMaxZero, and where scale * kDown stays in range
          simple_lane = simple_lane && __hbge2(zv, zero2) && __hble2(zv, max_zero2) && __hbeq2(__hsub2(__hadd2(zv, whole2), whole2), zv) &&
                        __hble2(__habs2(sd2[i][cb]), max_scale2);
        }
      }
      const bool simple = __all_sync(0xffffffffu, simple_lane);   // (both forms agree to the bit where both apply)
      if (it + kGroups < n_units) {
        fetch_advance();
        fetch();
      }
      if constexpr (C::kHalfStages) {   // (the stage is waited for where the first store needs it)
        if (!mbar_wait(wctx, bar_raw_full + 8 * sr, pr, 0x400u + sr)) break;
      } else {
        if (!mbar_wait_both(wctx, bar_raw_full + 8 * sr, pr, 0x400u + sr, bar_deq_empty + 8 * sd, pd ^ 1u, 0x480u + sd)) break;
      }
      bool ok = true;
      const uint32_t src = rawst_base + sr * kRawStageBytes + lane_off;
#pragma unroll
      for (int kh = 0; kh < C::kKHalves; ++kh) {
        uint32_t w[2][4];                // [32-k part][8-row block, block of 16 columns]
        ldmatrix_x4_trans(src + kh * (32 * 128), w[0]);
        ldmatrix_x4_trans(src + kh * (32 * 128) + 16 * 128, w[1]);
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          uint32_t cells[16];            // 64 k = 32 operand columns of this block's 16 weight columns
          if (simple) {
            const int r1 = FINE ? 1 : 0;
            const V2 s_lo[2] = {P16::low(sd2[0][cb]), P16::low(sd2[r1][cb])}, s_hi[2] = {P16::high(sd2[0][cb]), P16::high(sd2[r1][cb])};
            const V2 z_lo[2] = {P16::low(zd2[0][cb]), P16::low(zd2[r1][cb])}, z_hi[2] = {P16::high(zd2[0][cb]), P16::high(zd2[r1][cb])};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t w0 = w[q >> 1][2 * (q & 1) + cb];
              const uint32_t lo4 = w0 & 0x0F0F0F0Fu, hi4 = (w0 >> 4) & 0x0F0F0F0Fu;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                // byte i: column 2g + (i & 1), row 2s + (i >> 1); selector 8 + j replicates the sign of
                // byte j, which is zero
                const uint32_t sel = i | ((8 + i) << 4) | ((4 + i) << 8) | ((12 + i) << 12);
                const V2 x = P16::from_bits(byte_perm_sign(lo4, hi4, sel));
                const V2 z = (i & 1) ? z_hi[q >> 1] : z_lo[q >> 1], sx = (i & 1) ? s_hi[q >> 1] : s_lo[q >> 1];
                cells[4 * q + 2 * (i & 1) + (i >> 1)] = P16::bits(__hmul2(__hfma2(x, up2, z), sx));
              }
            }
          } else {
            // zero-points that are not small integers: the fp32 statement, verbatim
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t w0 = w[q >> 1][2 * (q & 1) + cb];
              const int r = FINE ? q >> 1 : 0;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t b8 = (w0 >> (8 * i)) & 0xFFu;
                const V2 sv = P16::from_bits(s_cur[r][cb]), zv = P16::from_bits(z_cur[r][cb]);
                const float z0 = (i & 1) ? P16::hi(zv) : P16::lo(zv);
                const float s0 = (i & 1) ? P16::hi(sv) : P16::lo(sv);
                cells[4 * q + 2 * (i & 1) + (i >> 1)] =
                    P16::bits(P16::make(__fmul_rn(__fsub_rn(static_cast<float>(b8 & 15u), z0), s0),
                                        __fmul_rn(__fsub_rn(static_cast<float>(b8 >> 4), z0), s0)));
              }
            }
          }
          if (C::kHalfStages && cb == 0) ok = mbar_wait(wctx, bar_deq_empty + 8 * sd, pd ^ 1u, 0x480u + sd);
          if (ok) tmem_st_16x256b(lane_dst + kh * 32 + sd * C::kDeqTmemCols + (static_cast<uint32_t>(16 * cb) << 16), cells);
        }
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_raw_empty + 8 * sr);   // every byte of the packed stage has been read
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_deq_full + 8 * sd);
    }
  } else if (warp >= 4 + kDeqWarps) {
    // -------------------------------- epilogue --------------------------------
    const int quarter = warp & 3;
    const int n_local = quarter * 32 + column_of_lane(lane);   // weight column inside the tile
    const int et = threadIdx.x - (128 + kDeqWarps * 32);
    // token columns of this warp: all of the tile, or one half of it
    const int half = (warp - (4 + kDeqWarps)) >> 2;
    const int cc_half = C::kEpiWarps == 4 ? p.mt : ((p.mt >> 1) + 15) & ~15;
    const int cc_begin = half * cc_half;
    const int cc_end = cc_begin + cc_half < p.mt ? cc_begin + cc_half : p.mt;
    grid_dependency_wait();
    T* c = static_cast<T*>(p.c);
    const T* bias = static_cast<const T*>(p.bias);
    const size_t slot_floats = static_cast<size_t>(p.mt) * kTileN;
    uint32_t seg = 0;
    long long u = u_begin;
    while (u < u_end) {
      const long long tile = u / p.k_steps;
      const int ntile = static_cast<int>(tile / p.m_tiles);
      const int m0 = static_cast<int>(tile - static_cast<long long>(ntile) * p.m_tiles) * p.mt;
      const long long tile_begin = tile * p.k_steps;
      const long long tile_end = tile_begin + p.k_steps;
      const long long seg_end = tile_end < u_end ? tile_end : u_end;
      const bool whole = (u == tile_begin) && (seg_end == tile_end);
      // the MMA issuers take alternate units of the CTA's run (or a half of every unit); in a one-unit
      // segment only one of them has written its accumulators
      bool issuer_has_units[C::kIssuers];
#pragma unroll
      for (int i = 0; i < C::kIssuers; ++i) {
        // units of the segment are it0 .. it0 + len - 1; issuer i owns those with it % kIssuers == i
        const long long it0 = u - u_begin, len = seg_end - u;
        const long long first = it0 + ((i - it0 % C::kIssuers) + C::kIssuers) % C::kIssuers;
        issuer_has_units[i] = C::kHalfStages || first < it0 + len;
      }
      const uint32_t buf = seg % C::kAccBufs, pacc = (seg / C::kAccBufs) & 1u;
      ++seg;
      // Where a partial segment goes. Cluster: this CTA's shared memory (the ring is idle once
      // the accumulators of its only segment are complete). Equal runs: a slot in scratch;
      // a CTA's run holds at most two partial segments, slot 2c if the tile began in an earlier
      // CTA and slot 2c + 1 if it begins in c. The tile's arrival counter is its first CTA's.
      const bool shared_in_cluster = p.cluster_s > 1;
      const bool local = whole || shared_in_cluster;
      const int first_cta = local ? 0 : cta_of_unit(units, ctas, tile_begin);
      const int last_cta = local ? 0 : cta_of_unit(units, ctas, tile_end - 1);
      const int parts = last_cta - first_cta + 1;
      auto slot_of = [&](int part) {
        return p.slots + static_cast<size_t>(2 * (first_cta + part) + (part == 0 ? 1 : 0)) * slot_floats;
      };
      unsigned int* counter = p.counters + first_cta;
      const int n = ntile * kTileN + n_local;
      const bool n_ok = n < p.n;
      const int cols_ok = p.n - (ntile * kTileN + quarter * 32);   // of this warp's 32 columns
      const float bias_v = (bias != nullptr && n_ok) ? to_f32<T>(bias[n]) : 0.f;
      T* c_warp = c + static_cast<size_t>(m0) * p.n + ntile * kTileN + quarter * 32;
      const bool begins_tile = u == tile_begin;
      u = seg_end;
      if (!mbar_wait_long(wctx, bar_acc_full + 8 * buf, pacc, 0x500u + buf)) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * (C::kAccs * MTMAX);
      float* slot = whole ? nullptr
                    : shared_in_cluster ? reinterpret_cast<float*>(base_ptr)
                                        : slot_of(begins_tile ? 0 : static_cast<int>(blockIdx.x) - first_cta);
      for (int cc = cc_begin; cc < cc_end; cc += 16) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll
        for (int acc = 0; acc < C::kAccs; ++acc) {
          if (C::kIssuers > 1 && !issuer_has_units[acc / C::kAccsPerIssuer]) continue;   // stale accumulators
          uint32_t r[16];
          tmem_ld(taddr + acc * MTMAX + cc, r);
          tmem_wait_ld(r);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
        }
        if (whole) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += bias_v;
          store_tokens16<T>(c_warp + static_cast<size_t>(cc) * p.n, p.n, v, lane, p.m - (m0 + cc), cols_ok,
                            p.c_vec != 0);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            reinterpret_cast<float4*>(slot)[((cc >> 2) + q) * kTileN + n_local] =
                make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_empty + 8 * buf);
      if (!local) {
        // publish the partial, then find out whether this CTA completes the tile
        __threadfence();
        named_barrier_sync(1, C::kEpiThreads);
        if (et == 0) {
          const unsigned int prev = atomicAdd(counter, 1u);
          *last_flag = (prev == static_cast<unsigned int>(parts - 1)) ? 1u : 0u;
          if (prev == static_cast<unsigned int>(parts - 1)) *counter = 0u;  // ready for the next launch
        }
        named_barrier_sync(1, C::kEpiThreads);
        if (*last_flag != 0u) {
          __threadfence();
          // sixteen rows at a time; the loads of a part are issued before any is consumed
          for (int cc = cc_begin; cc < cc_end && m0 + cc < p.m; cc += 16) {
            float sum[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] = 0.f;
#pragma unroll 2
            for (int q = 0; q < parts; ++q) {
              const float4* src = reinterpret_cast<const float4*>(slot_of(q)) + (cc >> 2) * kTileN + n_local;
              float4 v[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) v[j] = __ldcg(src + j * kTileN);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                sum[4 * j] += v[j].x;
                sum[4 * j + 1] += v[j].y;
                sum[4 * j + 2] += v[j].z;
                sum[4 * j + 3] += v[j].w;
              }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] += bias_v;
            store_tokens16<T>(c_warp + static_cast<size_t>(cc) * p.n, p.n, sum, lane, p.m - (m0 + cc), cols_ok,
                              p.c_vec != 0);
          }
        }
        named_barrier_sync(1, C::kEpiThreads);  // last_flag may be rewritten only after everyone has read it
      }
    }
  }

  if (p.cluster_s > 1) {
    // Every CTA holds the partial sums of its part of K in shared memory. The cluster's warps
    // share the (16 tokens x 32 columns) blocks of the tile, and add the parts in part order.
    static_assert(MTMAX * kTileN * 4 <= C::kRing, "the partial tile fits the ring");
    __syncwarp();
    cluster_sync();
    const int part = static_cast<int>(blockIdx.x) % p.cluster_s;
    const int tile = static_cast<int>(blockIdx.x) / p.cluster_s;
    const int ntile = tile / p.m_tiles, m0 = (tile - ntile * p.m_tiles) * p.mt;
    // Block by block from CTA to CTA. (A CTA's warps first left all reading to the first CTA or two:
    // K=2048 N=1024 M=128 with eight parts 14.6 us, now 10.6.)
    constexpr int kWarps = C::kThreads / 32;
    for (int i = warp * p.cluster_s + part; i < p.mt / 4; i += p.cluster_s * kWarps) {
      const int cc = (i >> 2) * 16, quarter = i & 3;
      if (m0 + cc >= p.m) continue;
      const int n_local = quarter * 32 + column_of_lane(lane), n = ntile * kTileN + n_local;
      const T* bias = static_cast<const T*>(p.bias);
      const uint32_t src = base + ((cc >> 2) * kTileN + n_local) * 16;
      float sum[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) sum[j] = 0.f;
      for (int q = 0; q < p.cluster_s; ++q) {
        const uint32_t peer = cluster_map_shared(src, q);
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = ld_shared_cluster_f4(peer + j * (kTileN * 16));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sum[4 * j] += v[j].x;
          sum[4 * j + 1] += v[j].y;
          sum[4 * j + 2] += v[j].z;
          sum[4 * j + 3] += v[j].w;
        }
      }
      const float bias_v = (bias != nullptr && n < p.n) ? to_f32<T>(bias[n]) : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) sum[j] += bias_v;
      store_tokens16<T>(static_cast<T*>(p.c) + static_cast<size_t>(m0 + cc) * p.n + ntile * kTileN + quarter * 32, p.n,
                        sum, lane, p.m - (m0 + cc), p.n - (ntile * kTileN + quarter * 32), p.c_vec != 0);
    }
    __syncwarp();
    cluster_sync();   // nobody reads this CTA's shared memory any more
  }

  // ------------------------------- teardown -------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <typename T, int MTMAX, bool FINE>
ks_status_t launch_t(const CUtensorMap& tm_w, const CUtensorMap& tm_a, const Params& p, int grid,
                     cudaStream_t stream) {
  using C = Cfg<MTMAX, FINE>;
  auto kernel = w4a16_umma_kernel<T, MTMAX, FINE>;
  static std::mutex mu;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
      if (e != cudaSuccess) return cuda_status(e, "ks_gemm_w4a16");
      attr_done[dev] = true;
    }
  }
  return cuda_status(launch_programmatic_cluster(kernel, static_cast<unsigned>(grid), static_cast<unsigned>(p.cluster_s), true,
                                                 C::kThreads, C::kSmemBytes, stream, tm_w, tm_a, p),
                     "ks_gemm_w4a16");
}

template <typename T, bool FINE>
ks_status_t launch_mt(int mtmax, const CUtensorMap& tm_w, const CUtensorMap& tm_a, const Params& p, int grid,
                      cudaStream_t stream) {
  switch (mtmax) {
    case 32: return launch_t<T, 32, FINE>(tm_w, tm_a, p, grid, stream);
    case 64: return launch_t<T, 64, FINE>(tm_w, tm_a, p, grid, stream);
    case 128: return launch_t<T, 128, FINE>(tm_w, tm_a, p, grid, stream);
    default: return launch_t<T, 192, FINE>(tm_w, tm_a, p, grid, stream);
  }
}

}  // namespace

bool w4a16_eligible(const W4A16Args& a) {
  if (a.k % kStepK != 0) return false;
  // one scale row per 128-k step, or a whole number of rows per step
  if (a.group_size % kStepK != 0 && a.group_size != 64 && a.group_size != 32) return false;
  if (a.n % 16 != 0) return false;                // 16-byte row pitch of the packed weight
  if (!aligned16(a.a) || !aligned16(a.b_packed) || !aligned16(a.scales)) return false;
  if (a.zeros != nullptr && !aligned16(a.zeros)) return false;
  if (a.m > (1 << 24) || a.n > (1 << 28) || a.k > (1 << 28)) return false;
  return tma_available();
}

namespace {

struct Geometry {
  int mt = 0, mtmax = 0, m_tiles = 0, n_tiles = 0, k_steps = 0, grid = 0;
  int cluster_s = 1;
  bool split = true;
  size_t counter_bytes = 0, slot_bytes = 0;
};

// Estimated times, in ns, fitted to 1091 shapes (N 1024..28672, K 1024..14336, 1 to 2048 rows, scale groups of
// 128, 64 and 32), each with every way below and up to five tile widths; the choice by them takes 1.3-1.5 % more
// than the best of those on average (with the constants that 8 units per CTA had given: 3.2-3.6 %).
// One unit (128 columns x 128 k) of a token tile of `mt` rows in a long run:
double unit_ns(int mt, bool fine) { return mt <= 32 && !fine ? 385.0 + 0.95 * mt : 430.0 + 1.15 * mt; }

// Token tiles, and how the units go to the CTAs: whichever finishes first by this estimate.
//   cluster    a tile's K range over S CTAs, which exchange partial sums through shared memory
//              (3 us with the second pipeline fill); needs all clusters resident at once
//   whole      runs of whole tiles: the last round may leave SMs idle
//   even runs  no SM idles, but a tile's last CTA reads the other parts from L2: 5 us for the
//              hand-over and 0.27 us per part and 16 token rows (two warps share that work in
//              192-row tiles). K=4096 N=4096 M=16: 11.8 us against 10.1 with clusters; K=14336 N=6144
//              M=16: 23.3 against 25.3
// Fewer token tiles mean fewer dequantisations of a weight; more of them, more tiles to deal out.
Geometry geometry_of(const W4A16Args& a) {
  Geometry g;
  const int sms = sm_count();
  const bool fine = a.group_size % kStepK != 0;
  g.n_tiles = static_cast<int>((a.n + kTileN - 1) / kTileN);
  g.k_steps = static_cast<int>((a.k / kStepK + 1) & ~int64_t(1));
  int64_t capacity[kMaxClusterSplit + 1];
  for (int s = 2; s <= kMaxClusterSplit; ++s) capacity[s] = cluster_capacity(s);
  double best = 0;
  auto offer = [&](double cost, int mt, int m_tiles, int cluster_s, bool split) {
    if (best != 0 && cost >= best) return;
    best = cost;
    g.mt = mt;
    g.m_tiles = m_tiles;
    g.cluster_s = cluster_s;
    g.split = split;
  };
  const int lo = static_cast<int>((a.m + 191) / 192), hi = static_cast<int>((a.m + 31) / 32);
  for (int want = lo; want <= hi && want < lo + 24; ++want) {
    const int mt = static_cast<int>(((a.m + want - 1) / want + 15) & ~int64_t(15));
    const int m_tiles = static_cast<int>((a.m + mt - 1) / mt);
    const long long tiles = static_cast<long long>(g.n_tiles) * m_tiles;
    const double unit = unit_ns(mt, fine);
    const double drain = mt * 19.0;   // a tile's accumulators to C
    offer(static_cast<double>((tiles + sms - 1) / sms) * (g.k_steps * unit + drain), mt, m_tiles, 1, false);
    for (int s = 2; s <= kMaxClusterSplit && 2 * s <= g.k_steps && tiles * s <= sms; ++s) {
      if (capacity[s] < tiles) break;
      offer(2.0 * ((g.k_steps / 2 + s - 1) / s) * unit + drain + 3000.0, mt, m_tiles, s, false);
    }
    const double per_cta = static_cast<double>(tiles) * g.k_steps / (tiles * g.k_steps < sms ? tiles * g.k_steps : sms);
    const double parts = g.k_steps / per_cta + 1.0;
    const int chunks = mt <= 128 ? mt / 16 : (mt + 31) / 32;
    offer(per_cta * unit + (per_cta / g.k_steps + 1.0) * drain + 5000.0 + 270.0 * chunks * parts, mt, m_tiles, 1, true);
  }
  g.mtmax = g.mt <= 32 ? 32 : (g.mt <= 64 ? 64 : (g.mt <= 128 ? 128 : 192));
  const long long tiles = static_cast<long long>(g.n_tiles) * g.m_tiles;
  const long long work = g.split ? tiles * g.k_steps : tiles;
  g.grid = g.cluster_s > 1 ? static_cast<int>(tiles * g.cluster_s) : static_cast<int>(work < sms ? work : sms);
  g.slot_bytes = g.split ? static_cast<size_t>(g.grid) * 2 * g.mt * kTileN * sizeof(float) : 0;
  g.counter_bytes = (static_cast<size_t>(g.grid) * sizeof(unsigned int) + 255) & ~size_t(255);
  return g;
}

// The same token tiles dealt out whole, which takes no slots.
Geometry in_whole_tiles(Geometry g) {
  if (!g.split) return g;
  g.split = false;
  const long long tiles = static_cast<long long>(g.n_tiles) * g.m_tiles;
  g.grid = static_cast<int>(tiles < sm_count() ? tiles : sm_count());
  g.slot_bytes = 0;
  return g;
}

// Encodes the tensor maps and enqueues the kernel on scratch memory the caller of this
// function has already obtained: the arrival counters (all zero on entry; the
// kernel leaves them zero) and the fp32 partial slots.
ks_status_t enqueue_w4a16(const W4A16Args& a, const Geometry& g, unsigned int* counters, float* slots,
                          unsigned int* fault_word, cudaStream_t stream) {
  const bool bf16 = a.dtype == KS_DTYPE_BF16;
  const CUtensorMapDataType dt16 = bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm_w, tm_a;
  {
    // two K-steps per box; a step past the end of K reads zeros
    const uint64_t dims[2] = {static_cast<uint64_t>(a.n), static_cast<uint64_t>(a.k / 2)};
    const uint64_t str[1] = {static_cast<uint64_t>(a.n)};
    const uint32_t box[2] = {static_cast<uint32_t>(kTileN), static_cast<uint32_t>(kStepK)};
    if (!tma_encode(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a.b_packed, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B))
      KSB_FAIL(KS_ERROR_INTERNAL, "ks_gemm_w4a16: tensor map for the packed weight rejected");
  }
  {
    // A[M,K] seen as [K/64][M][64]: a box brings one or both 64-k swizzle atoms of a K-step
    const uint64_t dims[3] = {64u, static_cast<uint64_t>(a.m), static_cast<uint64_t>(a.k / 64)};
    const uint64_t str[2] = {static_cast<uint64_t>(a.k) * 2, 128u};
    const uint32_t box[3] = {64u, static_cast<uint32_t>(g.mt), g.mtmax <= 128 ? 2u : 1u};
    if (!tma_encode(&tm_a, dt16, 3, a.a, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B))
      KSB_FAIL(KS_ERROR_INTERNAL, "ks_gemm_w4a16: tensor map for the activations rejected");
  }

  const bool fine = a.group_size % kStepK != 0;
  Params p;
  p.c = a.c;
  p.bias = a.bias;
  p.scales = a.scales;
  p.zeros = a.zeros;
  p.counters = counters;
  p.slots = slots;
  p.fault_word = fault_word;
  p.m = static_cast<int>(a.m);
  p.n = static_cast<int>(a.n);
  p.k = static_cast<int>(a.k);
  p.mt = g.mt;
  p.m_tiles = g.m_tiles;
  p.n_tiles = g.n_tiles;
  p.k_steps = g.k_steps;
  p.gs_steps = fine ? 1 : a.group_size / kStepK;
  p.sub_shift = a.group_size == 64 ? 1 : 0;
  p.groups = static_cast<int>(a.k / a.group_size);
  p.split = g.split ? 1 : 0;
  p.cluster_s = g.cluster_s;
  p.c_vec = (reinterpret_cast<uintptr_t>(a.c) & 7) == 0 ? 1 : 0;
  p.has_zeros = a.zeros != nullptr ? 1 : 0;
  const uint32_t fmt = bf16 ? 1u : 0u;
  // weights: K along the columns in tensor memory
  p.idesc = umma_instr_desc(fmt, fmt, 0u, 0u, 128u, static_cast<uint32_t>(g.mt));

  if (bf16)
    return fine ? launch_mt<__nv_bfloat16, true>(g.mtmax, tm_w, tm_a, p, g.grid, stream)
                : launch_mt<__nv_bfloat16, false>(g.mtmax, tm_w, tm_a, p, g.grid, stream);
  return fine ? launch_mt<__half, true>(g.mtmax, tm_w, tm_a, p, g.grid, stream)
              : launch_mt<__half, false>(g.mtmax, tm_w, tm_a, p, g.grid, stream);
}

}  // namespace

// Which fast kernel. The register-operand decode kernel feeds legacy mma.sync, whose rate on
// this part is about a tenth of tcgen05's. Up to 8 rows (one MMA per 16 x 16 weight block) its cheaper
// arithmetic wins on long runs of units (256 columns x 128 k): from about 9 per SM, with scale groups of 32 or
// 64, where the other kernel's arithmetic costs more, from 5. Its split-K fix-up grows with the parts per
// tile, 2 per SM and tile: with fewer than one tile per 8 SMs (N < 4864) it loses what it gains.
// From 9 rows it is ahead only with narrow groups on wide weights. us, decode kernel | tcgen05:
//   M=8  group 128  N=28672 K=4096 24.7 | 28.3   N=11008 K=4096 15.3 | 16.5   N=6144 K=8192 16.0 | 17.1
//                   N=11008 K=2048 12.6 | 10.0   N=4096 K=14336 20.0 | 18.4
//   M=8  group 64   N=11008 K=4096 16.5 | 19.0   N=4096 K=8192 13.7 | 15.7    N=11008 K=2048 13.3 | 12.1
//   M=16 group 128  N=28672 K=4096 30.0 | 28.3   N=11008 K=8192 26.6 | 23.5
//   M=16 group 64   N=28672 K=4096 32.0 | 35.4   N=11008 K=8192 28.1 | 29.1   N=4096 K=14336 27.2 | 22.6
// The caller can pin either kernel.
bool use_decode_kernel(const W4A16Args& a) {
  if (a.kernel == 1 || !decode::eligible(a)) return false;
  if (a.kernel == 2 || !w4a16_eligible(a)) return true;
  const long long sms = sm_count(), tiles = (a.n + 255) / 256, units = tiles * (a.k / 128);
  const bool fine = a.group_size % kStepK != 0;
  if (a.m <= 8) return fine ? units >= 5 * sms : units >= 9 * sms && 8 * tiles >= sms;
  return fine && a.m <= 16 && units >= 12 * sms && 4 * tiles >= sms;
}

ks_status_t launch_w4a16(const W4A16Args& a, cudaStream_t stream) {
  // Counters and slots are separate allocations: the counters must be zero whenever no
  // kernel is running, and a region that another shape used for partial sums is not.
  // The tcgen05 kernels can give up on a bounded wait and leave counters non-zero; when
  // the fault poll has reported such a launch on this device, every stream's counters are
  // cleared before their next use (stream_scratch_mark_dirty).
  const bool dec = use_decode_kernel(a);
  const Geometry g = dec ? Geometry{} : geometry_of(a);
  const decode::Geometry gd = dec ? decode::geometry_of(a) : decode::Geometry{};
  const size_t slot_bytes = dec ? gd.slot_bytes : g.slot_bytes;
  const size_t counter_bytes = dec ? gd.counter_bytes : g.counter_bytes;
  // Whole tiles and clusters share nothing through memory.
  if (!dec && !g.split) return enqueue_w4a16(a, g, nullptr, nullptr, kernel_fault_word(), stream);
  StreamScratch scratch(stream);
  // More than 128 rows, and scale groups of 32 or 64, run without scratch memory where there is none: a graph
  // that is captured on a stream without it, a device without room.
  const bool can_do_without = w4a16_eligible(a) && a.kernel != 2 && (a.m > 128 || a.group_size % kStepK != 0);
  float* slots = nullptr;
  unsigned int* counters = nullptr;
  if (!(can_do_without && (scratch.cold_capture(slot_bytes, 0) || scratch.cold_capture(counter_bytes, 1)))) {
    slots = static_cast<float*>(scratch.get(slot_bytes, 0));
    counters = static_cast<unsigned int*>(scratch.get(counter_bytes, 1));
  }
  if (can_do_without && (slots == nullptr || counters == nullptr))
    return enqueue_w4a16(a, in_whole_tiles(geometry_of(a)), nullptr, nullptr, kernel_fault_word(), stream);
  if (slots == nullptr || counters == nullptr)
    KSB_FAIL(KS_ERROR_OUT_OF_MEMORY, "ks_gemm_w4a16: workspace allocation failed");
  if (std::getenv("KS_B200_ENV_RELOAD") != nullptr && std::getenv("KS_B200_TEST_DIRTY_COUNTERS") != nullptr) {
    // test hook: what a launch that gave up half-way leaves behind, without any GPU fault:
    // garbage in the counters and the mark that the fault poll would have set
    cudaMemsetAsync(counters, 0xFF, stream_scratch_bytes(stream, 1), stream);
    stream_scratch_mark_dirty(1);
    counters = static_cast<unsigned int*>(scratch.get(counter_bytes, 1));
    if (counters == nullptr) KSB_FAIL(KS_ERROR_INTERNAL, "ks_gemm_w4a16: clearing the split-K counters");
  }
  if (dec) return decode::enqueue(a, gd, counters, slots, stream);
  return enqueue_w4a16(a, g, counters, slots, kernel_fault_word(), stream);
}

// ---------------------------------------------------------------------------
// Variant for callers that must not allocate: the split-K slots and counters
// live in a fixed array inside the library image instead of scratch memory
// obtained from the CUDA allocator.
//
// `g_static_scratch` below is a __device__ array. In host code its name only
// stands for the symbol: it is not an address a kernel may dereference. The
// device address is asked for once per device (with that device current) with
// cudaGetSymbolAddress, and that pointer is what the kernel receives.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kStaticScratchBytes = size_t(16) << 20;  // 16 MiB on every GPU that loads the library
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

std::mutex g_static_mutex;
void* g_static_ptr[64] = {};

// Device address of the array on the current device; resolved on the first
// call per device. No allocation is involved.
ks_status_t static_scratch_address(uint8_t** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e, "ks_gemm_w4a16_static_scratch");
  if (dev < 0 || dev >= 64)
    KSB_FAIL(KS_ERROR_INTERNAL, "ks_gemm_w4a16_static_scratch: device ordinal out of the supported range");
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess) return cuda_status(e, "ks_gemm_w4a16_static_scratch: cudaGetSymbolAddress");
    if (ptr == nullptr)
      KSB_FAIL(KS_ERROR_INTERNAL, "ks_gemm_w4a16_static_scratch: the scratch symbol resolved to a null address");
    g_static_ptr[dev] = ptr;
  }
  *out = static_cast<uint8_t*>(g_static_ptr[dev]);
  return KS_SUCCESS;
}

}  // namespace

// What the fixed array is held against. Which shapes the entry point takes is part of its contract and
// must not change with the choice of kernel or deal, so this is not what a launch uses, but a bound
// of its own: partial sums per (column tile, part of K in equal runs), tiles of all rows. Where the
// kernel or deal chosen needs more than the array holds, one that fits takes its place: whole tiles
// need nothing.
size_t nominal_scratch(const W4A16Args& a) {
  if (a.m > 128 || a.group_size % kStepK != 0) return 0;
  const long long sms = sm_count();
  if (decode::eligible(a) && (a.kernel == 2 || (a.kernel == 0 && a.m <= 16 && (a.n + 255) / 256 * (a.k / 128) >= 20 * sms))) {
    const decode::Geometry d = decode::geometry_of(a);
    return d.counter_bytes + d.slot_bytes;
  }
  const long long mt = (a.m + 15) & ~int64_t(15);
  const long long n_tiles = (a.n + kTileN - 1) / kTileN, k_steps = a.k / kStepK;
  const long long units = n_tiles * k_steps;
  const long long per_cta = units / (units < sms ? units : sms);   // shortest run
  const long long max_parts = (k_steps + per_cta - 1) / per_cta + 1;
  return static_cast<size_t>(n_tiles * max_parts * mt * kTileN) * sizeof(float) +
         ((static_cast<size_t>(n_tiles) * sizeof(unsigned int) + 255) & ~size_t(255));
}

size_t w4a16_static_scratch_capacity() { return kStaticScratchBytes; }

ks_status_t launch_w4a16_static(const W4A16Args& a, cudaStream_t stream) {
  bool dec = use_decode_kernel(a);
  const decode::Geometry gd = dec ? decode::geometry_of(a) : decode::Geometry{};
  size_t need = nominal_scratch(a);
  if (dec && gd.counter_bytes + gd.slot_bytes > kStaticScratchBytes) {
    if (a.kernel == 0 && w4a16_eligible(a)) dec = false;
    else need = gd.counter_bytes + gd.slot_bytes;
  }
  if (need > kStaticScratchBytes) {
    char msg[224];
    snprintf(msg, sizeof(msg),
             "ks_gemm_w4a16_static_scratch: this shape counts as %zu bytes of split-K scratch, the built-in array "
             "holds %zu; use ks_gemm_w4a16 or fewer rows per call",
             need, kStaticScratchBytes);
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, msg);
  }
  Geometry g = dec ? Geometry{} : geometry_of(a);
  if (g.split && g.counter_bytes + g.slot_bytes > kStaticScratchBytes) g = in_whole_tiles(g);
  const size_t counter_bytes = dec ? gd.counter_bytes : g.counter_bytes;
  uint8_t* scratch = nullptr;
  ks_status_t st = static_scratch_address(&scratch);
  if (st != KS_SUCCESS) return st;
  // The array keeps whatever the previous call left. The kernels require the
  // arrival counters to be zero on entry (a clean run leaves them so, an aborted
  // one may not, and another shape lays them out differently); the slots are
  // fully overwritten before being read.
  // (one step with the launch: another thread's call on the stream may put slots where these counters are)
  static std::mutex enqueue_mutex;
  std::lock_guard<std::mutex> hold(enqueue_mutex);
  cudaError_t e = cudaMemsetAsync(scratch, 0, counter_bytes, stream);
  if (e != cudaSuccess) return cuda_status(e, "ks_gemm_w4a16_static_scratch: cudaMemsetAsync");
  unsigned int* counters = reinterpret_cast<unsigned int*>(scratch);
  float* slots = reinterpret_cast<float*>(scratch + counter_bytes);
  if (dec) return decode::enqueue(a, gd, counters, slots, stream);
  // The word through which a tcgen05 kernel reports a bounded wait that ran out is a pinned
  // host allocation made by the first allocating entry point on the device; a process that
  // only ever calls this entry point runs the tcgen05 kernel without it (the decode kernel
  // has no such wait).
  return enqueue_w4a16(a, g, counters, slots, kernel_fault_word_if_ready(), stream);
}

}  // namespace sm100
}  // namespace ksb

