// RMSNorm, alone and fused with the 1 x 128 FP8 group quantizer that usually follows it in
// front of a block-scaled GEMM.
//
// Reference: ks_rms_norm (include/kernel_set/norm.h:16-19, kernels/src/norm/rms_norm.cu:19-42).
// The arithmetic follows the reference's torch statement of the op (benchmarks/bench.py:
// 877-879): the normalised value x * rsqrt(mean(x^2) + eps) is rounded to the storage type,
// then multiplied by the weight and rounded again (the reference kernel keeps the product in
// fp32 and rounds once; the two differ by at most one unit in the last place). The
// fused form rounds the normalised row to the input type exactly as the plain kernel writes
// it and quantizes those values exactly as ks_quantize_fp8_group reads them, so its codes and
// scales are bit-identical to the two calls run one after the other, without the 16-bit
// intermediate ever reaching memory (the row is read once and kept in registers).
//
// A CTA per row, a thread owns one or two 16-element segments of it (rows of at most 8192 elements), so eight
// consecutive lanes hold the eight segments of a quantisation group, the arrangement quant_segment_codes
// expects. Issue-bound rather than memory-bound, so warps without segments are left out, and the
// products with the weight are taken two to an instruction: the normalised values and the weight are 16-bit,
// their product is exact in fp32, so the packed multiplication rounds once, as the scalar one did.
// Cold, event to event, with the quantizer, bf16: [4096,7168] 29.2 us, [4096,4096] 19.1, [16384,2048] 29.3 (128 threads
// with up to four segments and scalar products: 36.6, 23.0, 40.0).
#include <algorithm>
#include <string>

#include "common.cuh"
#include "kernel_set/norm.h"
#include "quant_math.cuh"
#include "sm100_host.cuh"
#include "sm100_ptx.cuh"

namespace ksb {
namespace {

using namespace quantmath;

constexpr int kNormThreads = 128;      // of the kernel for any width
constexpr int kMaxRowThreads = 256;
constexpr int kMaxSegs = 2;            // per thread
constexpr int kChains = 128;           // of a row's sum of squares

// A row's sum of squares has one order, whatever the number of threads, since a last place of it decides how some
// values of the row round: 128 chains, of which chain c adds up elements in turn (the kernel for any width: c, c + 128, ...;
// the other: segments c, c + 128, c + 256, c + 384), 32 chains to a warp, then the four warps' sums in pairs.
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// add(i, sum) adds a thread's i-th segment to a chain. With 128 threads and more the second segment continues the
// first one's chain, with fewer it is a chain of its own.
template <typename Add>
__device__ __forceinline__ float row_sum(const Add& add) {
  __shared__ float red[kChains / 32];
  __shared__ float handed[kChains];
  const int t = threadIdx.x, nt = blockDim.x, warp = t >> 5;
  if (nt < kChains) {
    const float a = warp_sum(add(0, 0.f)), b = warp_sum(add(1, 0.f));
    if ((t & 31) == 0) {
      red[warp] = a;
      red[warp + nt / 32] = b;
    }
    __syncthreads();
    return nt == 32 ? red[0] + red[1] : (red[0] + red[1]) + (red[2] + red[3]);
  }
  float v = 0.f;
  if (t < kChains) v = add(1, add(0, 0.f));
  if (nt > kChains) {
    // chain c goes on in thread c + 128
    if (t < kChains) handed[t] = v;
    __syncthreads();
    if (t >= kChains) v = add(1, add(0, handed[t - kChains]));
  }
  if (t >= kChains || t + kChains >= nt) {   // (whole warps)
    v = warp_sum(v);
    if ((t & 31) == 0) red[warp & 3] = v;
  }
  __syncthreads();
  return (red[0] + red[1]) + (red[2] + red[3]);
}

// y = (v * inv).to(T) * w, rounded to T: 16 elements. f32 needs no rounding in between.
__device__ __forceinline__ void scale_row(float (&v)[16], float inv, const Raw16<float>& w, uint4 (&y)[4]) {
  float g[16];
  w.unpack(g);
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = (v[j] * inv) * g[j];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    y[q] = make_uint4(__float_as_uint(v[4 * q]), __float_as_uint(v[4 * q + 1]), __float_as_uint(v[4 * q + 2]),
                      __float_as_uint(v[4 * q + 3]));
}
template <typename T>
__device__ __forceinline__ void scale_row(float (&v)[16], float inv, const Raw16<T>& w, uint4 (&y)[2]) {
  const uint32_t g[8] = {w.a.x, w.a.y, w.a.z, w.a.w, w.b.x, w.b.y, w.b.z, w.b.w};
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if constexpr (__is_same(T, __half)) {
      const __half2 n = __floats2half2_rn(v[2 * j] * inv, v[2 * j + 1] * inv);
      const __half2 p = __hmul2_rn(n, *reinterpret_cast<const __half2*>(&g[j]));
      o[j] = *reinterpret_cast<const uint32_t*>(&p);
    } else {
      const __nv_bfloat162 n = __floats2bfloat162_rn(v[2 * j] * inv, v[2 * j + 1] * inv);
      const __nv_bfloat162 p = __hmul2_rn(n, *reinterpret_cast<const __nv_bfloat162*>(&g[j]));
      o[j] = *reinterpret_cast<const uint32_t*>(&p);
    }
  }
  y[0] = make_uint4(o[0], o[1], o[2], o[3]);
  y[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// QUANT == false: out is T [rows, cols]. QUANT == true: out is fp8 [rows, cols], scale [rows, cols / 128].
template <typename T, bool QUANT, bool E5M2>
__global__ void __launch_bounds__(kMaxRowThreads)
rms_norm_rows_kernel(void* __restrict__ out, float* __restrict__ scale, const T* __restrict__ in,
                     const T* __restrict__ weight, int64_t cols, float eps, float qmax) {
  sm100::grid_dependency_wait();
  if constexpr (QUANT) sm100::grid_launch_dependents();
  const int64_t row = blockIdx.x;
  const int segs = static_cast<int>(cols / 16);
  const T* x = in + row * cols;
  // threads 0-127 own segments t and t + 128 (up to 64 threads: t and t + 64 or 32), the others those 256 further on
  const int first = threadIdx.x + (threadIdx.x & kChains), step = blockDim.x < kChains ? blockDim.x : kChains;
  Raw16<T> raw[kMaxSegs];
#pragma unroll
  for (int i = 0; i < kMaxSegs; ++i) {
    const int seg = first + i * step;
    raw[i] = seg < segs ? Raw16<T>::load(x + seg * 16) : Raw16<T>::zero();
  }
  const float sumsq = row_sum([&](int i, float sum) {
    float v[16];
    raw[i].unpack(v);
#pragma unroll
    for (int j = 0; j < 16; ++j) sum = fmaf(v[j], v[j], sum);
    return sum;
  });
  const float inv_rms = rsqrtf(sumsq / static_cast<float>(cols) + eps);
#pragma unroll
  for (int i = 0; i < kMaxSegs; ++i) {
    const int seg = first + i * step;
    const bool live = seg < segs;
    if (!__any_sync(0xffffffffu, live)) break;
    float v[16];
    raw[i].unpack(v);
    uint4 y[sizeof(T)];
    scale_row(v, inv_rms, live ? Raw16<T>::load(weight + seg * 16) : Raw16<T>::zero(), y);
    if constexpr (QUANT) {
      Raw16<T> r;
      r.a = y[0];
      r.b = y[1];
      r.unpack(v);
      float sc;
      const uint4 codes = quant_segment_codes<E5M2>(v, qmax, &sc);
      if (live) {
        if ((threadIdx.x & 7) == 0) scale[row * (cols / 128) + (seg >> 3)] = sc;
        __stcs(reinterpret_cast<uint4*>(static_cast<uint8_t*>(out) + row * cols + seg * 16), codes);
      }
    } else if (live) {
      uint4* dst = reinterpret_cast<uint4*>(static_cast<T*>(out) + row * cols + seg * 16);
#pragma unroll
      for (int q = 0; q < static_cast<int>(sizeof(T)); ++q) dst[q] = y[q];
    }
  }
}

// Any width / alignment: one CTA per row, the row read twice.
template <typename T>
__global__ void __launch_bounds__(kNormThreads)
rms_norm_any_kernel(T* __restrict__ out, const T* __restrict__ in, const T* __restrict__ weight, int64_t cols,
                    float eps) {
  sm100::grid_dependency_wait();
  const int64_t row = blockIdx.x;
  const T* x = in + row * cols;
  const float sumsq = row_sum([&](int i, float sum) {
    if (i > 0) return sum;
    for (int64_t c = threadIdx.x; c < cols; c += kNormThreads) {
      const float v = to_f32<T>(x[c]);
      sum = fmaf(v, v, sum);
    }
    return sum;
  });
  const float inv_rms = rsqrtf(sumsq / static_cast<float>(cols) + eps);
  for (int64_t c = threadIdx.x; c < cols; c += kNormThreads)
    out[row * cols + c] = from_f32<T>(to_f32<T>(from_f32<T>(to_f32<T>(x[c]) * inv_rms)) * to_f32<T>(weight[c]));
}

// Threads for a row, in whole warps: two segments to a thread, the 256 segments behind the first 256 to threads of their own.
unsigned row_threads(int64_t cols) {
  const unsigned segs = static_cast<unsigned>(cols / 16);
  if (segs <= kChains) return (segs + 63) / 64 * 32;
  if (segs <= 2 * kChains) return kChains;
  return kChains + std::min<unsigned>(kChains, (segs - 2 * kChains + 31) / 32 * 32);
}

bool rows_kernel_fits(int64_t cols, const void* a, const void* b, const void* c) {
  return cols % 128 == 0 && cols <= 16 * kMaxRowThreads * kMaxSegs && aligned16(a) && aligned16(b) &&
         aligned16(c);
}

}  // namespace
}  // namespace ksb

using namespace ksb;

extern "C" ks_status_t ks_rms_norm(void* out, const void* input, const void* weight, int64_t rows, int64_t cols,
                                   float eps, ks_dtype_t dtype, ks_stream_t stream) {
  const char* where = "ks_rms_norm";
  KSB_REQUIRE_PTR(out);
  KSB_REQUIRE_PTR(input);
  KSB_REQUIRE_PTR(weight);
  if (rows < 0 || cols <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_rms_norm: bad shape");
  if (!is_float3(dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_rms_norm: unsupported dtype");
  if (rows == 0) return KS_SUCCESS;
  if (rows > 2147483647LL) KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_rms_norm: grid exceeds CUDA grid limits");
  ks_status_t st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const unsigned grid = static_cast<unsigned>(rows);
  const bool fast = rows_kernel_fits(cols, out, input, weight);
#define KSB_RN(T)                                                                                               \
  do {                                                                                                          \
    if (fast) sm100::launch_programmatic(rms_norm_rows_kernel<T, false, false>, grid, row_threads(cols), 0, s, \
        out, nullptr, static_cast<const T*>(input), static_cast<const T*>(weight), cols, eps, 0.f);             \
    else sm100::launch_programmatic(rms_norm_any_kernel<T>, grid, kNormThreads, 0, s, \
        static_cast<T*>(out), static_cast<const T*>(input), \
                                                              static_cast<const T*>(weight), cols, eps);        \
  } while (0)
  if (dtype == KS_DTYPE_F32) KSB_RN(float);
  else if (dtype == KS_DTYPE_F16) KSB_RN(__half);
  else KSB_RN(__nv_bfloat16);
#undef KSB_RN
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}

extern "C" ks_status_t ks_rms_norm_quant_fp8(void* out_fp8, float* out_scale, const void* input, const void* weight,
                                             int64_t rows, int64_t cols, float eps, ks_dtype_t in_dtype,
                                             ks_dtype_t fp8_dtype, ks_stream_t stream) {
  const char* where = "ks_rms_norm_quant_fp8";
  KSB_REQUIRE_PTR(out_fp8);
  KSB_REQUIRE_PTR(out_scale);
  KSB_REQUIRE_PTR(input);
  KSB_REQUIRE_PTR(weight);
  if (rows < 0 || cols <= 0) KSB_FAIL(KS_ERROR_INVALID_ARGUMENT, "ks_rms_norm_quant_fp8: bad shape");
  if (!rows_kernel_fits(cols, out_fp8, input, weight))
    KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE,
             "ks_rms_norm_quant_fp8: cols must be a multiple of 128, at most 8192, and the buffers 16-byte aligned");
  if (!is_fp8(fp8_dtype)) KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_rms_norm_quant_fp8: fp8_dtype must be e4m3 or e5m2");
  if (in_dtype != KS_DTYPE_F16 && in_dtype != KS_DTYPE_BF16)
    KSB_FAIL(KS_ERROR_UNSUPPORTED_DTYPE, "ks_rms_norm_quant_fp8: input must be f16 or bf16");
  if (rows == 0) return KS_SUCCESS;
  if (rows > 2147483647LL) KSB_FAIL(KS_ERROR_UNSUPPORTED_SHAPE, "ks_rms_norm_quant_fp8: grid exceeds CUDA grid limits");
  ks_status_t st = require_sm100(where);
  if (st != KS_SUCCESS) return st;
  cudaStream_t s = as_stream(stream);
  const unsigned grid = static_cast<unsigned>(rows);
  const bool e5 = fp8_dtype == KS_DTYPE_F8E5M2;
#define KSB_RQ(T)                                                                                                 \
  do {                                                                                                            \
    if (e5) sm100::launch_programmatic(rms_norm_rows_kernel<T, true, true>, grid, row_threads(cols), 0, s, \
        out_fp8, out_scale, static_cast<const T*>(input), static_cast<const T*>(weight), cols, eps, 57344.0f);    \
    else sm100::launch_programmatic(rms_norm_rows_kernel<T, true, false>, grid, row_threads(cols), 0, s, \
        out_fp8, out_scale, static_cast<const T*>(input), static_cast<const T*>(weight), cols, eps, 448.0f);      \
  } while (0)
  if (in_dtype == KS_DTYPE_F16) KSB_RQ(__half);
  else KSB_RQ(__nv_bfloat16);
#undef KSB_RQ
  KSB_CHECK_LAUNCH(where);
  return KS_SUCCESS;
}
