// The steps of a mixture-of-experts layer that sit between the router's logits and the
// two grouped expert GEMMs, and after them: gate (softmax + top-k), the permutation that
// sorts (token, slot) pairs by expert, the row gather (optionally fused with the 1 x 128
// FP8 quantizer), SwiGLU between the GEMMs (optionally fused with the re-quantisation),
// and the weighted sum that brings expert outputs back to token order.
//
// Reference: ks_moe_gate_softmax_topk (kernels/src/moe/moe_gate.cu:43-119),
// ks_moe_compute_permutation / ks_moe_permute / ks_moe_unpermute
// (kernels/src/moe/moe_permute.cu:60-170, 179-380), ks_swiglu / ks_swiglu_packed
// (kernels/src/activation/gated_mlp.cu:39-134). Differences, on purpose:
//   * nothing here allocates per call or synchronises the stream (the reference's
//     permutation and unpermute launchers cudaMalloc, cudaStreamSynchronize and cudaFree
//     on every call, moe_permute.cu:205-242, 317-375); the one piece of workspace, the
//     inverse permutation of ks_moe_unpermute, is a stream-ordered library buffer;
//   * the permutation is a STABLE counting sort (pairs of one expert keep their
//     token order), so results are reproducible; the reference scatters with atomics and
//     leaves the order inside an expert unspecified;
//   * the gate evaluates exp with expf (the reference's torch statement, benchmarks/
//     bench.py:1555-1557, is the parity target; the reference kernel uses __expf).
#include <cstdio>
#include <type_traits>

#include <mutex>

#include "common.cuh"
#include "kernel_set/activation.h"
#include "kernel_set/moe.h"
#include "quant_math.cuh"
#include "sm100_host.cuh"
#include "sm100_ptx.cuh"

namespace ksb {
namespace {

constexpr int kMaxExperts = 1024;   // as the reference (moe_gate.cu:33)
constexpr int kMaxTopK = 32;        // as the reference (moe_gate.cu:35)

// ---------------------------------------------------------------------------------
// gate: one warp per token
// ---------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
gate_softmax_topk_kernel(float* __restrict__ out_w, int32_t* __restrict__ out_i, const T* __restrict__ logits,
                         int64_t tokens, int experts, int top_k, int renorm) {
  sm100::grid_start();
  extern __shared__ float gate_smem[];   // [warps][experts]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t token = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + warp;
  if (token >= tokens) return;   // whole warp
  float* p = gate_smem + warp * experts;
  const T* row = logits + token * experts;
  float mx = -3.4028235e38f;
  for (int e = lane; e < experts; e += 32) {
    const float v = to_f32<T>(row[e]);
    p[e] = v;
    mx = fmaxf(mx, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
  for (int e = lane; e < experts; e += 32) {
    const float ex = expf(p[e] - mx);
    p[e] = ex;
    sum += ex;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  for (int e = lane; e < experts; e += 32) p[e] = __fdiv_rn(p[e], sum);
  __syncwarp();
  // top-k by repeated arg-max; among equal probabilities the lowest expert id wins
  float my_w = 0.f;
  int my_i = 0;
  float chosen_sum = 0.f;
  for (int k = 0; k < top_k; ++k) {
    float best = -1.f;
    int best_e = 0x7fffffff;
    for (int e = lane; e < experts; e += 32) {
      const float v = p[e];
      if (v > best) { best = v; best_e = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
      if (ov > best || (ov == best && oe < best_e)) { best = ov; best_e = oe; }
    }
    if (lane == k) { my_w = best; my_i = best_e; }
    chosen_sum += best;
    if (lane == 0 && best_e < experts) p[best_e] = -2.f;   // not selectable again
    __syncwarp();
  }
  if (lane < top_k) {
    out_w[token * top_k + lane] = renorm ? __fdiv_rn(my_w, chosen_sum) : my_w;
    out_i[token * top_k + lane] = my_i;
  }
}

// ---------------------------------------------------------------------------------
// permutation: stable counting sort of the pairs by expert, no workspace
// ---------------------------------------------------------------------------------
// CTA b places the pairs of chunk b. It needs, per expert, the number of pairs in all chunks
// (where an expert's rows begin) and in the chunks before its own (where its pairs go in
// there). Every CTA counts all of that for itself: the ids are 4 bytes a pair and come
// from L2, so reading them once per CTA costs less than handing counts from CTA to CTA would (a second
// launch or a grid-wide wait). Inside a chunk, warp w owns a contiguous piece and walks it 32
// pairs at a time: position = running counter of (warp, expert) + number of lower lanes
// with the same expert in this step, which keeps the sort stable.
constexpr int kPermThreads = 1024;
constexpr int kPermWarps = kPermThreads / 32;

// Adds the pairs [begin, end) to the warp's row of `cnt`. Loads are issued eight at a time.
__device__ __forceinline__ void count_pairs(int* mine, const int32_t* __restrict__ topk_idx, int64_t begin,
                                            int64_t end, int experts) {
  for (int64_t base = begin + threadIdx.x; base < end; base += 8 * kPermThreads) {
    int e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t i = base + static_cast<int64_t>(j) * kPermThreads;
      e[j] = i < end ? __ldg(topk_idx + i) : -1;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (e[j] >= 0 && e[j] < experts) atomicAdd(mine + e[j], 1);
  }
}

// Sums `cnt` over the warps into `sum` and clears it.
__device__ __forceinline__ void fold_counts(int* cnt, int* sum, int experts) {
  __syncthreads();
  for (int e = threadIdx.x; e < experts; e += kPermThreads) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < kPermWarps; ++w) {
      run += cnt[w * experts + e];
      cnt[w * experts + e] = 0;
    }
    sum[e] = run;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kPermThreads)
compute_permutation_kernel(int32_t* __restrict__ sorted_ids, int32_t* __restrict__ offsets,
                           const int32_t* __restrict__ topk_idx, int64_t pairs, int experts, int64_t chunk) {
  sm100::grid_start();
  extern __shared__ int perm_smem[];       // [warps][experts] counters, then two [experts] rows
  int* cnt = perm_smem;
  int* before = perm_smem + kPermWarps * experts;   // pairs of an expert in the chunks before this one
  int* total = before + experts;                    // ... in the chunks after it, then in all
  __shared__ int warp_sums[kPermWarps];
  __shared__ int routed_pairs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t c_begin = static_cast<int64_t>(blockIdx.x) * chunk;
  const int64_t c_end = c_begin + chunk < pairs ? c_begin + chunk : pairs;
  // this CTA's pairs: a piece of chunk / 32 (a multiple of 32) per warp, in the first `warps` warps
  const int64_t piece = chunk / kPermWarps;
  const int64_t begin = c_begin + warp * piece;
  const int64_t end = begin + piece < c_end ? begin + piece : c_end;
  const int warps = static_cast<int>((c_end - c_begin + piece - 1) / piece);
  // the ids of a warp's first step stay in registers: with up to 1024 pairs a CTA that is all of them
  const int e_first = begin + lane < end ? __ldg(topk_idx + begin + lane) : -1;
  const int rows = gridDim.x == 1 ? warps : kPermWarps;   // of `cnt` in use
  for (int i = threadIdx.x; i < rows * experts; i += kPermThreads) cnt[i] = 0;
  for (int i = threadIdx.x; i < 2 * experts; i += kPermThreads) before[i] = 0;
  __syncthreads();
  int* mine = cnt + warp * experts;
  if (c_begin > 0) {
    count_pairs(mine, topk_idx, 0, c_begin, experts);
    fold_counts(cnt, before, experts);
  }
  if (c_end < pairs) {
    count_pairs(mine, topk_idx, c_end, pairs, experts);
    fold_counts(cnt, total, experts);
  }
  for (int64_t base = begin; base < end; base += 32) {
    const int64_t i = base + lane;
    const int e = base == begin ? e_first : (i < end ? __ldg(topk_idx + i) : -1);
    const bool valid = e >= 0 && e < experts;
    const unsigned mask = __match_any_sync(0xffffffffu, valid ? e : experts + lane);
    if (valid && lane == __ffs(mask) - 1) mine[e] += __popc(mask);
    __syncwarp();
  }
  __syncthreads();
  // exclusive scan over warps for every expert, starting behind the earlier chunks
  for (int e = threadIdx.x; e < experts; e += kPermThreads) {
    int run = before[e];
#pragma unroll 8
    for (int w = 0; w < warps; ++w) {
      const int c = cnt[w * experts + e];
      cnt[w * experts + e] = run;
      run += c;
    }
    total[e] += run;
  }
  __syncthreads();
  // exclusive scan of the totals over experts (experts <= 1024 = one element per thread)
  {
    const int v = threadIdx.x < experts ? total[threadIdx.x] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const int ws = warp_sums[lane];
      int winc = ws;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, winc, o);
        if (lane >= o) winc += t;
      }
      warp_sums[lane] = winc - ws;
    }
    __syncthreads();
    const int excl = inc - v + warp_sums[warp];
    if (threadIdx.x < experts) {
      total[threadIdx.x] = excl;
      if (blockIdx.x == 0) offsets[threadIdx.x] = excl;
      if (threadIdx.x == experts - 1) {
        routed_pairs = excl + v;
        if (blockIdx.x == 0) offsets[experts] = excl + v;
      }
    }
  }
  __syncthreads();
  for (int64_t base = begin; base < end; base += 32) {
    const int64_t i = base + lane;
    const int e = base == begin ? e_first : (i < end ? __ldg(topk_idx + i) : -1);
    const bool valid = e >= 0 && e < experts;
    const unsigned mask = __match_any_sync(0xffffffffu, valid ? e : experts + lane);
    if (valid) sorted_ids[total[e] + mine[e] + __popc(mask & ((1u << lane) - 1u))] = static_cast<int32_t>(i);
    __syncwarp();
    if (valid && lane == __ffs(mask) - 1) mine[e] += __popc(mask);
    __syncwarp();
  }
  // pairs with an expert id out of range are dropped; their places at the end hold -1
  for (int64_t i = routed_pairs + static_cast<int64_t>(blockIdx.x) * kPermThreads + threadIdx.x; i < pairs;
       i += static_cast<int64_t>(gridDim.x) * kPermThreads)
    sorted_ids[i] = -1;
}

// ---------------------------------------------------------------------------------
// permute: gather token rows into expert order
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
permute_rows16_kernel(uint4* __restrict__ out, const uint4* __restrict__ in, const int32_t* __restrict__ ids,
                      int64_t pairs, int top_k, int64_t row_vec) {
  sm100::grid_dependency_wait();
  const int64_t total = pairs * row_vec;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = t / row_vec, c = t - r * row_vec;
    const int32_t pair = __ldg(ids + r);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (pair >= 0 && pair < pairs) v = __ldg(in + static_cast<int64_t>(pair / top_k) * row_vec + c);
    __stcs(out + t, v);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
permute_rows_any_kernel(T* __restrict__ out, const T* __restrict__ in, const int32_t* __restrict__ ids,
                        int64_t pairs, int top_k, int64_t hidden) {
  sm100::grid_dependency_wait();
  const int64_t total = pairs * hidden;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = t / hidden, c = t - r * hidden;
    const int32_t pair = ids[r];
    out[t] = (pair >= 0 && pair < pairs) ? in[static_cast<int64_t>(pair / top_k) * hidden + c] : from_f32<T>(0.f);
  }
}

// Gather fused with the 1 x 128 quantizer: output row r holds the codes of token
// ids[r] / top_k; a lane owns 16 elements, 8 lanes a group (as quant_group128_kernel).
template <typename T, bool E5M2>
__global__ void __launch_bounds__(256)
permute_quant_kernel(uint8_t* __restrict__ out, float* __restrict__ scale, const T* __restrict__ in,
                     const int32_t* __restrict__ ids, int64_t pairs, int top_k, int64_t hidden, float qmax) {
  sm100::grid_start();
  const int64_t segs_per_row = hidden / 16;
  const int64_t seg = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t r = seg / segs_per_row;
  const bool live = r < pairs;
  float v[16];
  bool have = false;
  if (live) {
    const int32_t pair = __ldg(ids + r);
    if (pair >= 0 && pair < pairs) {
      quantmath::Vec16<T>::load(in + static_cast<int64_t>(pair / top_k) * hidden + (seg - r * segs_per_row) * 16, v);
      have = true;
    }
  }
  if (!have) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.f;
  }
  quantmath::quant_segment<T, E5M2>(out, scale, v, seg, live, qmax);
}

// ---------------------------------------------------------------------------------
// unpermute: out[token] = sum_k w[token, k] * permuted[row of pair (token, k)]
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
inverse_permutation_kernel(int32_t* __restrict__ inverse, const int32_t* __restrict__ ids, int64_t pairs) {
  sm100::grid_start();
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= pairs) return;
  const int32_t pair = ids[r];
  if (pair >= 0 && pair < pairs) inverse[pair] = static_cast<int32_t>(r);
}

// `row` if it is the row of pair `pair`, else -1.
__device__ __forceinline__ int32_t check_row(int32_t row, const int32_t* __restrict__ ids, int64_t pair, int64_t pairs) {
  return (row >= 0 && row < pairs && __ldg(ids + row) == pair) ? row : -1;
}

// Row of a pair after the sort, -1 for a dropped pair. The inverse map of a dropped pair was not
// written by this call and holds whatever an earlier one left there, so the row it names is
// looked up again: only the row that really holds the pair counts. (Clearing the map first was
// a launch of its own.)
__device__ __forceinline__ int32_t row_of_pair(const int32_t* __restrict__ inverse, const int32_t* __restrict__ ids,
                                               int64_t pair, int64_t pairs) {
  return check_row(__ldg(inverse + pair), ids, pair, pairs);
}

// permute_quant_kernel the other way round, for large problems: a token is read and quantized
// once and its codes are written to the rows of all its pairs. (Row by row, every row quantizes its token
// again: 145 instructions per 512 elements, top_k times, made that the bound: 141 us for 4096
// tokens x 7168 x top 8, where writing the 242 MB takes ~40.) Blocks from `token_blocks` on walk the rows and
// do those that no token's inverse entry names: ids out of range (a row of zeros) and
// repeated ids, which the row-by-row kernel takes as they come. With experts on other ranks most ids are
// out of range, so such rows have a warp each and are written without the quantizer's arithmetic:
// the shape above with 7/8 dropped 106 us row by row, 285 with 32 rows to a warp and the arithmetic, 68 now.
// With two or three pairs a token it also pays to look whether the token has a row at all before it is read
// (`look_first`): 16384 tokens x 4096, top 2, all dropped 55 us row by row, 75 without, 45 with; f32 with none
// dropped 106 us row by row, 79 without, 85 with.
template <typename T, bool E5M2>
__global__ void __launch_bounds__(256)
permute_quant_tokens_kernel(uint8_t* __restrict__ out, float* __restrict__ scale, const T* __restrict__ in,
                            const int32_t* __restrict__ ids, const int32_t* __restrict__ inverse, int64_t tokens,
                            int top_k, int64_t hidden, unsigned token_blocks, bool look_first, float qmax) {
  sm100::grid_start();
  const int64_t segs_per_row = hidden / 16;
  const int64_t pairs = tokens * top_k;
  float v[16];
  if (blockIdx.x < token_blocks) {
    const int64_t seg = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t token = seg / segs_per_row;
    const int64_t c = seg - token * segs_per_row;
    bool live = token < tokens;
    if (look_first) {
      // a token without rows, all its experts elsewhere, is not even read
      bool named = false;
      for (int k = 0; k < top_k && !named && live; ++k) named = row_of_pair(inverse, ids, token * top_k + k, pairs) >= 0;
      live = named;
      if (!__any_sync(0xffffffffu, live)) return;
    }
    if (live) {
      quantmath::Vec16<T>::load(in + token * hidden + c * 16, v);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
    }
    float sc;
    const uint4 codes = quantmath::quant_segment_codes<E5M2>(v, qmax, &sc);
    if (!live) return;
    for (int k = 0; k < top_k; ++k) {
      const int32_t row = row_of_pair(inverse, ids, token * top_k + k, pairs);
      if (row < 0) continue;
      const int64_t dst = row * segs_per_row + c;
      if ((c & 7) == 0) scale[dst >> 3] = sc;
      __stcs(reinterpret_cast<uint4*>(out + dst * 16), codes);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t r = (static_cast<int64_t>(blockIdx.x - token_blocks) * blockDim.x + threadIdx.x) >> 5;   // this warp's row
  if (r >= pairs) return;
  const int32_t pair = __ldg(ids + r);
  if (pair < 0 || pair >= pairs) {   // what the quantizer makes of a row of zeros
    for (int64_t c = lane; c < segs_per_row; c += 32) {
      const int64_t dst = r * segs_per_row + c;
      if ((c & 7) == 0) scale[dst >> 3] = quantmath::kScaleFloor;
      __stcs(reinterpret_cast<uint4*>(out + dst * 16), make_uint4(0u, 0u, 0u, 0u));
    }
    return;
  }
  if (__ldg(inverse + pair) == r) return;
  for (int64_t c0 = 0; c0 < segs_per_row; c0 += 32) {   // (segs_per_row is a multiple of 8)
    const int64_t c = c0 + lane;
    const bool live = c < segs_per_row;
    if (live) {
      quantmath::Vec16<T>::load(in + static_cast<int64_t>(pair / top_k) * hidden + c * 16, v);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
    }
    quantmath::quant_segment<T, E5M2>(out, scale, v, r * segs_per_row + c, live, qmax);
  }
}

// A thread owns 8 consecutive columns (16 bytes of a 16-bit type) of one token; slots are
// added in slot order in fp32 and the row is written once.
template <typename T>
__global__ void __launch_bounds__(256)
unpermute_vec8_kernel(T* __restrict__ out, const T* __restrict__ permuted, const int32_t* __restrict__ inverse,
                      const int32_t* __restrict__ ids,
                      const float* __restrict__ weights, int64_t tokens, int top_k, int64_t hidden) {
  sm100::grid_dependency_wait();
  const int64_t row_vec = hidden / 8;
  const int64_t total = tokens * row_vec;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t token = t / row_vec, c = t - token * row_vec;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    // four slots at a time: their index loads, then their rows, are in flight together (one slot
    // after the other is a chain of three loads per slot)
    for (int k0 = 0; k0 < top_k; k0 += 4) {
      int32_t prow[4];
      float w[4];
      uint4 raw[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool in = k0 + j < top_k;
        prow[j] = in ? __ldg(inverse + token * top_k + k0 + j) : -1;
        w[j] = in ? __ldg(weights + token * top_k + k0 + j) : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) prow[j] = check_row(prow[j], ids, token * top_k + k0 + j, tokens * top_k);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (prow[j] >= 0)
          raw[j] = __ldcs(reinterpret_cast<const uint4*>(permuted + static_cast<int64_t>(prow[j]) * hidden) + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (prow[j] < 0) continue;
        const T* x = reinterpret_cast<const T*>(&raw[j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(to_f32<T>(x[i]), w[j], acc[i]);
      }
    }
    uint4 o;
    T* y = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = from_f32<T>(acc[j]);
    *(reinterpret_cast<uint4*>(out + token * hidden) + c) = o;
  }
}

// The same an element at a time, from a map that was cleared first (-1: dropped). Looking every row up again,
// as above, is one more dependent load per element and slot here: 4096 tokens x 7168, top 8, f32 297 us
// with the clearing launch, 613 with the look-up.
template <typename T>
__global__ void __launch_bounds__(256)
unpermute_any_kernel(T* __restrict__ out, const T* __restrict__ permuted, const int32_t* __restrict__ inverse,
                     const float* __restrict__ weights, int64_t tokens, int top_k, int64_t hidden) {
  sm100::grid_dependency_wait();
  const int64_t total = tokens * hidden;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t token = t / hidden, c = t - token * hidden;
    float acc = 0.f;
    for (int k = 0; k < top_k; ++k) {
      const int32_t prow = inverse[token * top_k + k];
      if (prow < 0) continue;
      acc = fmaf(to_f32<T>(permuted[static_cast<int64_t>(prow) * hidden + c]), weights[token * top_k + k], acc);
    }
    out[t] = from_f32<T>(acc);
  }
}

// ---------------------------------------------------------------------------------
// SwiGLU
// ---------------------------------------------------------------------------------
__device__ __forceinline__ float silu(float x) { return __fdiv_rn(x, 1.0f + expf(-x)); }

// Two 16-bit values in a word: as fp32, and from fp32.
template <typename T>
__device__ __forceinline__ float2 unpack_pair(uint32_t w) {
  if constexpr (__is_same(T, __half)) return __half22float2(*reinterpret_cast<const __half2*>(&w));
  else return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (__is_same(T, __half)) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
// |both| < 64 (false with a NaN).
template <typename T>
__device__ __forceinline__ bool below_64(uint32_t w) {
  constexpr uint32_t k64 = __is_same(T, __half) ? 0x5400u : 0x4280u;
  return (w & 0x7fffu) < k64 && ((w >> 16) & 0x7fffu) < k64;
}

// y = silu(g) * u, rounded to T, for 16 elements in words of two; g is replaced. These kernels are bound by
// their instructions, most of which the IEEE division took (with its test for operands that need scaling):
// for |g| < 64 the divisor lies in [1, 7e27] and the quotient is far from overflow, so the
// approximate reciprocal and one correction step (Markstein: q0 = g * r, q = q0 + (g - q0 * d) * r, the residual
// exact in an FMA) do, two to an instruction. On sm_100 the result is the rounded quotient for every 16-bit gate
// (tested over all of them), so it does not matter which way an element's neighbours, or the address of its row,
// send it. Anything else, infinities and NaN with it, is divided. 32768 x 2048 with the quantizer 100 -> 82 us cold.
template <typename T>
__device__ __forceinline__ void silu_mul_16(uint32_t (&g)[8], const uint32_t (&u)[8]) {
  using namespace quantmath;
  bool small = true;
#pragma unroll
  for (int i = 0; i < 8; ++i) small = small && below_64<T>(g[i]);
  if (small) {
    const F2 one = pack2(1.f, 1.f), neg1 = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 gf = unpack_pair<T>(g[i]), uf = unpack_pair<T>(u[i]);
      const F2 x = pack2(gf.x, gf.y);
      const F2 d = fma2(pack2(expf(-gf.x), expf(-gf.y)), one, one);
      float d0, d1, r0, r1, y0, y1;
      unpack2(d, &d0, &d1);
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
      const F2 r = pack2(r0, r1);
      const F2 q0 = mul2(x, r);
      const F2 e = fma2(q0, d, mul2(x, neg1));   // q0 * d - x
      unpack2(mul2(fma2(e, mul2(r, neg1), q0), pack2(uf.x, uf.y)), &y0, &y1);
      g[i] = pack_pair<T>(y0, y1);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 gf = unpack_pair<T>(g[i]), uf = unpack_pair<T>(u[i]);
      g[i] = pack_pair<T>(silu(gf.x) * uf.x, silu(gf.y) * uf.y);
    }
  }
}
template <typename T>
__device__ __forceinline__ void load_words(const T* p, uint32_t (&w)[8]) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

// out[r, c] = silu(gate[r, c]) * up[r, c]; gate and up are rows of `in_stride` elements
// starting at gate0 / up0 (packed: gate0 = in, up0 = in + inter, stride 2 * inter).
template <typename T>
__global__ void __launch_bounds__(256)
swiglu_kernel(T* __restrict__ out, const T* __restrict__ gate0, const T* __restrict__ up0, int64_t rows,
              int64_t inter, int64_t in_stride) {
  sm100::grid_dependency_wait();
  const int64_t total = rows * inter;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = t / inter, c = t - r * inter;
    out[t] = from_f32<T>(silu(to_f32<T>(gate0[r * in_stride + c])) * to_f32<T>(up0[r * in_stride + c]));
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
swiglu_vec16_kernel(T* __restrict__ out, const T* __restrict__ gate0, const T* __restrict__ up0, int64_t rows,
                    int64_t inter, int64_t in_stride) {
  sm100::grid_dependency_wait();
  const int64_t segs_per_row = inter / 16;
  const int64_t seg = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t r = seg / segs_per_row;
  if (r >= rows) return;
  const int64_t c = (seg - r * segs_per_row) * 16;
  uint32_t g[8], u[8];
  load_words(gate0 + r * in_stride + c, g);
  load_words(up0 + r * in_stride + c, u);
  silu_mul_16<T>(g, u);
  uint4* dst = reinterpret_cast<uint4*>(out + r * inter + c);
  dst[0] = make_uint4(g[0], g[1], g[2], g[3]);
  dst[1] = make_uint4(g[4], g[5], g[6], g[7]);
}

// Packed SwiGLU fused with the 1 x 128 quantizer: the activation is rounded to T exactly
// as the unfused kernel writes it, then quantized exactly as the quantizer reads it.
template <typename T, bool E5M2>
__global__ void __launch_bounds__(256)
swiglu_quant_kernel(uint8_t* __restrict__ out, float* __restrict__ scale, const T* __restrict__ in, int64_t rows,
                    int64_t inter, float qmax) {
  sm100::grid_start();
  const int64_t segs_per_row = inter / 16;
  const int64_t seg = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t r = seg / segs_per_row;
  const bool live = r < rows;
  float v[16];
  if (live) {
    const int64_t c = (seg - r * segs_per_row) * 16;
    uint32_t g[8], u[8];
    load_words(in + r * 2 * inter + c, g);
    load_words(in + r * 2 * inter + inter + c, u);
    silu_mul_16<T>(g, u);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 f = unpack_pair<T>(g[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.f;
  }
  quantmath::quant_segment<T, E5M2>(out, scale, v, seg, live, qmax);
}

inline unsigned grid_for(int64_t work_items, int threads = 256) {
  const int64_t blocks = (work_items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(sm_count()) * 16;
  return static_cast<unsigned>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

ks_status_t check_pairs(const char* where, int64_t tokens, int top_k, int64_t* pairs) {
  if (tokens > 0 && top_k > 0 && tokens > INT32_MAX / top_k)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, std::string(where) + ": num_tokens*top_k exceeds int32 limit");
  *pairs = tokens * static_cast<int64_t>(top_k);
  return KS_SUCCESS;
}

}  // namespace
}  // namespace ksb

using namespace ksb;

namespace {
template <typename T>
void launch_swiglu(void* out, const void* gate, const void* up, int64_t rows, int64_t inter, int64_t stride,
                   cudaStream_t s) {
  const bool vec = !std::is_same<T, float>::value && inter % 16 == 0 && stride % 8 == 0 && aligned16(out) &&
                   aligned16(gate) && aligned16(up);
  if (vec) {
    const int64_t segs = rows * (inter / 16);
    sm100::launch_programmatic(swiglu_vec16_kernel<T>, static_cast<unsigned>((segs + 255) / 256), 256, 0, s,
        static_cast<T*>(out), static_cast<const T*>(gate), static_cast<const T*>(up), rows, inter, stride);
  } else {
    sm100::launch_programmatic(swiglu_kernel<T>, grid_for(rows * inter), 256, 0, s,
        static_cast<T*>(out), static_cast<const T*>(gate),
                                                            static_cast<const T*>(up), rows, inter, stride);
  }
}

ks_status_t swiglu_common(const char* where, void* out, const void* gate, const void* up, int64_t rows,
                          int64_t inter, int64_t stride, ks_dtype_t dtype, ks_stream_t stream) {
  if (rows < 0 || inter <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, std::string(where) + ": bad shape");
  if (!is_float3(dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, std::string(where) + ": unsupported dtype");
  if (rows == 0) return KS_SUCCESS;
  if (rows * (inter / 16 + 1) / 256 > 2147483647LL)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, std::string(where) + ": grid exceeds CUDA grid limits");
  ks_status_t st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  if (dtype == KS_DTYPE_F32) launch_swiglu<float>(out, gate, up, rows, inter, stride, s);
  else if (dtype == KS_DTYPE_F16) launch_swiglu<__half>(out, gate, up, rows, inter, stride, s);
  else launch_swiglu<__nv_bfloat16>(out, gate, up, rows, inter, stride, s);
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}
}  // namespace

extern "C" {

ks_status_t ks_moe_gate_softmax_topk(float* out_weights, int32_t* out_indices, const void* logits,
                                     int64_t num_tokens, int num_experts, int top_k, int renormalize,
                                     ks_dtype_t dtype, ks_stream_t stream) {
  const char* where = "ks_moe_gate_softmax_topk";
  KSB_REQUIRE_PTR(out_weights);
  KSB_REQUIRE_PTR(out_indices);
  KSB_REQUIRE_PTR(logits);
  if (num_tokens < 0 || num_experts <= 0 || top_k <= 0 || top_k > num_experts)
    KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_moe_gate_softmax_topk: bad shape");
  if (num_experts > kMaxExperts || top_k > kMaxTopK)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_moe_gate_softmax_topk: at most 1024 experts and top_k 32");
  if (!is_float3(dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_moe_gate_softmax_topk: unsupported dtype");
  if (num_tokens == 0) return KS_SUCCESS;
  ks_status_t st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const int warps = num_experts <= 256 ? 8 : 2;   // 8 KB of shared memory per CTA either way
  const unsigned blocks = static_cast<unsigned>((num_tokens + warps - 1) / warps);
  const size_t smem = static_cast<size_t>(warps) * num_experts * sizeof(float);
#define KSB_GATE(T)                                                                                          \
  sm100::launch_programmatic(gate_softmax_topk_kernel<T>, blocks, warps * 32, smem, s, \
      out_weights, out_indices, \
                                                               static_cast<const T*>(logits), num_tokens,   \
                                                               num_experts, top_k, renormalize)
  if (dtype == KS_DTYPE_F32) KSB_GATE(float);
  else if (dtype == KS_DTYPE_F16) KSB_GATE(__half);
  else KSB_GATE(__nv_bfloat16);
#undef KSB_GATE
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

ks_status_t ks_moe_compute_permutation(int32_t* sorted_token_ids, int32_t* expert_offsets,
                                       const int32_t* topk_indices, int64_t num_tokens, int num_experts,
                                       int top_k, ks_stream_t stream) {
  const char* where = "ks_moe_compute_permutation";
  KSB_REQUIRE_PTR(sorted_token_ids);
  KSB_REQUIRE_PTR(expert_offsets);
  KSB_REQUIRE_PTR(topk_indices);
  if (num_tokens < 0 || num_experts <= 0 || top_k <= 0)
    KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_moe_compute_permutation: bad shape");
  if (num_experts > kMaxExperts)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_moe_compute_permutation: at most 1024 experts");
  int64_t pairs = 0;
  ks_status_t st = check_pairs(where, num_tokens, top_k, &pairs);
  if (st != KS_SUCCESS) return st;
  st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const size_t smem = (static_cast<size_t>(kPermWarps) + 2) * num_experts * sizeof(int);
  // one pair per thread, at most one CTA per SM
  const int64_t per_cta = (pairs + sm_count() - 1) / sm_count();
  const int64_t per_thread = (per_cta + kPermThreads - 1) / kPermThreads;
  const int64_t chunk = (per_thread > 0 ? per_thread : 1) * kPermThreads;
  const unsigned ctas = pairs > 0 ? static_cast<unsigned>((pairs + chunk - 1) / chunk) : 1u;
  // once per device and always: the kernel's static shared memory counts towards the 48 KB that need no
  // opt-in, so a test of the dynamic part alone left out 361 experts (49096 + 132 bytes)
  static std::mutex mu;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(compute_permutation_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>((kPermWarps + 2) * kMaxExperts * sizeof(int)));
      if (e != cudaSuccess) return cuda_status(e, where);
      attr_done[dev] = true;
    }
  }
  sm100::launch_programmatic(compute_permutation_kernel, ctas, kPermThreads, smem, s,
      sorted_token_ids, expert_offsets, topk_indices, pairs,
                                                              num_experts, chunk);
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

ks_status_t ks_moe_permute(void* permuted, const void* input, const int32_t* sorted_token_ids, int64_t num_tokens,
                           int top_k, int64_t hidden, ks_dtype_t dtype, ks_stream_t stream) {
  const char* where = "ks_moe_permute";
  KSB_REQUIRE_PTR(permuted);
  KSB_REQUIRE_PTR(input);
  KSB_REQUIRE_PTR(sorted_token_ids);
  if (num_tokens < 0 || top_k <= 0 || hidden <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_moe_permute: bad shape");
  if (!is_float3(dtype) && !is_fp8(dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_moe_permute: unsupported dtype");
  int64_t pairs = 0;
  ks_status_t st = check_pairs(where, num_tokens, top_k, &pairs);
  if (st != KS_SUCCESS) return st;
  if (pairs == 0) return KS_SUCCESS;
  st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const int64_t elt = dtype == KS_DTYPE_F32 ? 4 : (is_fp8(dtype) ? 1 : 2);
  const int64_t row_bytes = hidden * elt;
  if (row_bytes % 16 == 0 && aligned16(permuted) && aligned16(input)) {
    const int64_t row_vec = row_bytes / 16;
    sm100::launch_programmatic(permute_rows16_kernel, grid_for(pairs * row_vec), 256, 0, s,
        static_cast<uint4*>(permuted), static_cast<const uint4*>(input), sorted_token_ids, pairs, top_k, row_vec);
  } else if (elt == 4) {
    sm100::launch_programmatic(permute_rows_any_kernel<float>, grid_for(pairs * hidden), 256, 0, s,
        static_cast<float*>(permuted), static_cast<const float*>(input), sorted_token_ids, pairs, top_k, hidden);
  } else if (elt == 2) {
    sm100::launch_programmatic(permute_rows_any_kernel<__half>, grid_for(pairs * hidden), 256, 0, s,
        static_cast<__half*>(permuted), static_cast<const __half*>(input), sorted_token_ids, pairs, top_k, hidden);
  } else {
    sm100::launch_programmatic(permute_rows_any_kernel<__nv_fp8_e4m3>, grid_for(pairs * hidden), 256, 0, s,
        static_cast<__nv_fp8_e4m3*>(permuted), static_cast<const __nv_fp8_e4m3*>(input), sorted_token_ids, pairs,
        top_k, hidden);
  }
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

ks_status_t ks_moe_permute_quant_fp8(void* out_fp8, float* out_scale, const void* input,
                                     const int32_t* sorted_token_ids, int64_t num_tokens, int top_k,
                                     int64_t hidden, ks_dtype_t in_dtype, ks_dtype_t fp8_dtype,
                                     ks_stream_t stream) {
  const char* where = "ks_moe_permute_quant_fp8";
  KSB_REQUIRE_PTR(out_fp8);
  KSB_REQUIRE_PTR(out_scale);
  KSB_REQUIRE_PTR(input);
  KSB_REQUIRE_PTR(sorted_token_ids);
  if (num_tokens < 0 || top_k <= 0 || hidden <= 0)
    KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_moe_permute_quant_fp8: bad shape");
  if (hidden % 128 != 0 || !aligned16(out_fp8) || !aligned16(input))
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE,
             "ks_moe_permute_quant_fp8: hidden must be a multiple of 128 and the buffers 16-byte aligned");
  if (!is_fp8(fp8_dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_moe_permute_quant_fp8: fp8_dtype must be e4m3 or e5m2");
  if (!is_float3(in_dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_moe_permute_quant_fp8: unsupported dtype");
  int64_t pairs = 0;
  ks_status_t st = check_pairs(where, num_tokens, top_k, &pairs);
  if (st != KS_SUCCESS) return st;
  if (pairs == 0) return KS_SUCCESS;
  st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const int64_t segs = pairs * (hidden / 16);
  if ((segs + 255) / 256 > 2147483647LL)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_moe_permute_quant_fp8: grid exceeds CUDA grid limits");
  const unsigned blocks = static_cast<unsigned>((segs + 255) / 256);
  const bool e5 = fp8_dtype == KS_DTYPE_F8E5M2;
  uint8_t* o = static_cast<uint8_t*>(out_fp8);
  // Token by token where the quantizing that it saves outweighs the extra launch (the inverse map,
  // ~2.5 us), also with most pairs dropped, where row by row has little to do: from 24 M elements with six
  // pairs a token, 32 M with four, 64 M with two. us, row by row | token by token, none and all dropped:
  //   1024 x 6 x 4096 16.5 | 14.0, 12.4 | 12.4    512 x 8 x 4096 12.4 | 11.4, 10.3 | 11.2 (stays row by row)
  //   4096 x 4 x 4096 41.0 | 23.2, 28.8 | 25.4    2400 x 4 x 2048 14.4 | 12.0, 10.4 | 12.4 (stays)
  //   16384 x 2 x 4096 88 | 68, 55 | 45           4096 x 2 x 7168 38.8 | 33.4, half dropped 30.9 | 34.1 (stays)
  // The map lives in stream scratch; a stream under capture, where scratch may not grow, keeps to rows.
  const int64_t token_route_from = int64_t(top_k >= 6 ? 24 : top_k >= 4 ? 32 : 64) << 20;
  if (top_k >= 2 && pairs * hidden >= token_route_from) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess) {
      cudaGetLastError();
      capturing = cudaStreamCaptureStatusActive;
    }
    sm100::StreamScratch scratch(s);   // (until both kernels are enqueued)
    int32_t* inverse = capturing != cudaStreamCaptureStatusNone
                           ? nullptr
                           : static_cast<int32_t*>(scratch.get(static_cast<size_t>(pairs) * sizeof(int32_t), 4));
    if (inverse != nullptr) {
      sm100::launch_programmatic(inverse_permutation_kernel, static_cast<unsigned>((pairs + 255) / 256), 256, 0, s,
          inverse, sorted_token_ids, pairs);
      const unsigned token_blocks = static_cast<unsigned>((num_tokens * (hidden / 16) + 255) / 256);
      const unsigned total_blocks = token_blocks + static_cast<unsigned>((pairs + 7) / 8);
#define KSB_PT(T, E5, QMAX)                                                                                      \
  sm100::launch_programmatic(permute_quant_tokens_kernel<T, E5>, total_blocks, 256, 0, s, \
      o, out_scale, static_cast<const T*>(input), \
                                                                  sorted_token_ids, inverse, num_tokens, top_k,  \
                                                                  hidden, token_blocks, top_k < 4, QMAX)
      if (in_dtype == KS_DTYPE_F32) { if (e5) KSB_PT(float, true, 57344.0f); else KSB_PT(float, false, 448.0f); }
      else if (in_dtype == KS_DTYPE_F16) { if (e5) KSB_PT(__half, true, 57344.0f); else KSB_PT(__half, false, 448.0f); }
      else { if (e5) KSB_PT(__nv_bfloat16, true, 57344.0f); else KSB_PT(__nv_bfloat16, false, 448.0f); }
#undef KSB_PT
      KSB_CHECK_LAUNCH(where);
      return KS_SUCCESS;
    }
  }
#define KSB_PQ(T)                                                                                               \
  do {                                                                                                          \
    if (e5) sm100::launch_programmatic(permute_quant_kernel<T, true>, blocks, 256, 0, s, \
        o, out_scale, static_cast<const T*>(input), \
                                                                 sorted_token_ids, pairs, top_k, hidden, 57344.0f); \
    else sm100::launch_programmatic(permute_quant_kernel<T, false>, blocks, 256, 0, s, \
        o, out_scale, static_cast<const T*>(input), \
                                                               sorted_token_ids, pairs, top_k, hidden, 448.0f); \
  } while (0)
  if (in_dtype == KS_DTYPE_F32) KSB_PQ(float);
  else if (in_dtype == KS_DTYPE_F16) KSB_PQ(__half);
  else KSB_PQ(__nv_bfloat16);
#undef KSB_PQ
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

ks_status_t ks_moe_unpermute(void* out, const void* permuted, const int32_t* sorted_token_ids,
                             const float* routing_weights, int64_t num_tokens, int top_k, int64_t hidden,
                             ks_dtype_t dtype, ks_stream_t stream) {
  const char* where = "ks_moe_unpermute";
  KSB_REQUIRE_PTR(out);
  KSB_REQUIRE_PTR(permuted);
  KSB_REQUIRE_PTR(sorted_token_ids);
  KSB_REQUIRE_PTR(routing_weights);
  if (num_tokens < 0 || top_k <= 0 || hidden <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_moe_unpermute: bad shape");
  if (!is_float3(dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_moe_unpermute: unsupported dtype");
  int64_t pairs = 0;
  ks_status_t st = check_pairs(where, num_tokens, top_k, &pairs);
  if (st != KS_SUCCESS) return st;
  if (pairs == 0) return KS_SUCCESS;
  st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  // inverse[pair] = row of the pair after the sort (not written for dropped pairs). Stream-ordered
  // library workspace: allocated when the stream first needs it (or needs more), never freed
  // or synchronised per call.
  sm100::StreamScratch scratch(s);   // (until both kernels are enqueued)
  int32_t* inverse = static_cast<int32_t*>(scratch.get(static_cast<size_t>(pairs) * sizeof(int32_t), 4));
  if (inverse == nullptr) KSB_FAIL(KS_ERROR_OUT_OF_MEMORY, "ks_moe_unpermute: workspace allocation failed");
  const bool vec = dtype != KS_DTYPE_F32 && hidden % 8 == 0 && aligned16(out) && aligned16(permuted);
  if (!vec) {
    const cudaError_t e = cudaMemsetAsync(inverse, 0xFF, static_cast<size_t>(pairs) * sizeof(int32_t), s);
    if (e != cudaSuccess) return cuda_status(e, where);
  }
  sm100::launch_programmatic(inverse_permutation_kernel, static_cast<unsigned>((pairs + 255) / 256), 256, 0, s,
      inverse, sorted_token_ids, pairs);
#define KSB_UNPERMUTE(T)                                                                                           \
  do {                                                                                                             \
    T* o = static_cast<T*>(out);                                                                                   \
    const T* x = static_cast<const T*>(permuted);                                                                  \
    if (vec) sm100::launch_programmatic(unpermute_vec8_kernel<T>, grid_for(num_tokens * (hidden / 8)), 256, 0, s, \
        o, x, inverse, sorted_token_ids, routing_weights, num_tokens, top_k, hidden);                              \
    else sm100::launch_programmatic(unpermute_any_kernel<T>, grid_for(num_tokens * hidden), 256, 0, s, \
        o, x, inverse, routing_weights, \
                                                                               num_tokens, top_k, hidden);         \
  } while (0)
  if (dtype == KS_DTYPE_F32) sm100::launch_programmatic(unpermute_any_kernel<float>,
      grid_for(num_tokens * hidden), 256, 0, s,
      static_cast<float*>(out), static_cast<const float*>(permuted), inverse, routing_weights, num_tokens, top_k, hidden);
  else if (dtype == KS_DTYPE_F16) KSB_UNPERMUTE(__half);
  else KSB_UNPERMUTE(__nv_bfloat16);
#undef KSB_UNPERMUTE
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

ks_status_t ks_swiglu(void* out, const void* gate, const void* up, int64_t rows, int64_t inter, ks_dtype_t dtype,
                      ks_stream_t stream) {
  KSB_REQUIRE_PTR(out);
  KSB_REQUIRE_PTR(gate);
  KSB_REQUIRE_PTR(up);
  return swiglu_common("ks_swiglu", out, gate, up, rows, inter, inter, dtype, stream);
}

ks_status_t ks_swiglu_packed(void* out, const void* input, int64_t rows, int64_t inter, ks_dtype_t dtype,
                             ks_stream_t stream) {
  KSB_REQUIRE_PTR(out);
  KSB_REQUIRE_PTR(input);
  if (inter <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_swiglu_packed: bad shape");
  const int64_t elt = dtype == KS_DTYPE_F32 ? 4 : 2;
  const void* up = static_cast<const uint8_t*>(input) + inter * elt;
  return swiglu_common("ks_swiglu_packed", out, input, up, rows, inter, 2 * inter, dtype, stream);
}

ks_status_t ks_swiglu_packed_quant_fp8(void* out_fp8, float* out_scale, const void* input, int64_t rows,
                                       int64_t inter, ks_dtype_t in_dtype, ks_dtype_t fp8_dtype,
                                       ks_stream_t stream) {
  const char* where = "ks_swiglu_packed_quant_fp8";
  KSB_REQUIRE_PTR(out_fp8);
  KSB_REQUIRE_PTR(out_scale);
  KSB_REQUIRE_PTR(input);
  if (rows < 0 || inter <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_swiglu_packed_quant_fp8: bad shape");
  if (inter % 128 != 0 || !aligned16(out_fp8) || !aligned16(input))
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE,
             "ks_swiglu_packed_quant_fp8: inter must be a multiple of 128 and the buffers 16-byte aligned");
  if (!is_fp8(fp8_dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_swiglu_packed_quant_fp8: fp8_dtype must be e4m3 or e5m2");
  if (in_dtype != KS_DTYPE_F16 && in_dtype != KS_DTYPE_BF16)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_swiglu_packed_quant_fp8: input must be f16 or bf16");
  if (rows == 0) return KS_SUCCESS;
  ks_status_t st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const int64_t segs = rows * (inter / 16);
  if ((segs + 255) / 256 > 2147483647LL)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_swiglu_packed_quant_fp8: grid exceeds CUDA grid limits");
  const unsigned blocks = static_cast<unsigned>((segs + 255) / 256);
  const bool e5 = fp8_dtype == KS_DTYPE_F8E5M2;
  uint8_t* o = static_cast<uint8_t*>(out_fp8);
#define KSB_SQ(T)                                                                                                    \
  do {                                                                                                               \
    if (e5) sm100::launch_programmatic(swiglu_quant_kernel<T, true>, blocks, 256, 0, s, \
        o, out_scale, static_cast<const T*>(input), rows, \
                                                                inter, 57344.0f);                                    \
    else sm100::launch_programmatic(swiglu_quant_kernel<T, false>, blocks, 256, 0, s, \
        o, out_scale, static_cast<const T*>(input), rows, \
                                                              inter, 448.0f);                                        \
  } while (0)
  if (in_dtype == KS_DTYPE_F16) KSB_SQ(__half);
  else KSB_SQ(__nv_bfloat16);
#undef KSB_SQ
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

}  // extern "C"
