#include "sm100_host.cuh"

#include <cstdlib>

#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace ksb {
namespace sm100 {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
    cudaGetLastError();
  });
  return fn;
}

struct Scratch {
  void* ptr = nullptr;
  size_t bytes = 0;
  bool dirty = false;
  bool in_graph = false;         // a captured graph holds the address
  std::vector<void*> retired;    // buffers that graphs hold and that have been outgrown
};
__global__ void __launch_bounds__(256) full_sm_kernel() {}   // only asked about, never launched

std::mutex g_scratch_mutex;
std::map<std::pair<std::pair<int, cudaStream_t>, int>, Scratch> g_scratch;

}  // namespace

bool tma_available() { return encode_fn() != nullptr; }

bool tma_encode(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base, const uint64_t* dims,
                const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr || rank < 2 || rank > 3) return false;
  cuuint64_t gdim[3];
  cuuint64_t gstr[2];
  cuuint32_t bdim[3];
  cuuint32_t estr[3] = {1, 1, 1};
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
  }
  for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides_bytes[i];
  return fn(map, dtype, static_cast<cuuint32_t>(rank), const_cast<void*>(base), gdim, gstr, bdim, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

StreamScratch::StreamScratch(cudaStream_t stream) : stream_(stream) {
  if (cudaGetDevice(&dev_) != cudaSuccess) {
    dev_ = -1;
    return;
  }
  // a lock per (device, stream), out of a fixed set: streams that share one wait for each other's
  // launches, a few microseconds of host time
  static std::mutex locks[64];
  const uintptr_t h = reinterpret_cast<uintptr_t>(stream) / 16 + static_cast<uintptr_t>(dev_) * 7;
  lock_ = std::unique_lock<std::mutex>(locks[(h ^ (h >> 6) ^ (h >> 12)) % 64]);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();
    status = cudaStreamCaptureStatusActive;
  }
  capturing_ = status != cudaStreamCaptureStatusNone;
}

StreamScratch::~StreamScratch() {
  for (int i = 0; i < owned_count_; ++i)
    if (cudaFreeAsync(owned_[i], stream_) != cudaSuccess) cudaGetLastError();
}

bool StreamScratch::cold_capture(size_t bytes, int kind) const {
  return capturing_ && stream_scratch_bytes(stream_, kind) < bytes;
}

namespace {

void* zeroed(size_t bytes, cudaStream_t stream) {
  void* fresh = nullptr;
  if (cudaMallocAsync(&fresh, bytes, stream) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (cudaMemsetAsync(fresh, 0, bytes, stream) != cudaSuccess) {
    cudaGetLastError();
    cudaFreeAsync(fresh, stream);
    return nullptr;
  }
  return fresh;
}

}  // namespace

void* StreamScratch::get(size_t bytes, int kind) {
  if (dev_ < 0) return nullptr;
  const size_t floor_bytes = kind == 0 ? (size_t(1) << 20) : (size_t(64) << 10);
  size_t want = bytes < floor_bytes ? floor_bytes : bytes;
  want = (want + 0xFFFF) & ~size_t(0xFFFF);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  Scratch& s = g_scratch[std::make_pair(std::make_pair(dev_, stream_), kind)];
  if (s.bytes >= bytes && s.ptr != nullptr) {
    if (s.dirty) {
      if (cudaMemsetAsync(s.ptr, 0, s.bytes, stream_) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
      }
      s.dirty = capturing_;   // a captured clearing has not happened yet
    }
    s.in_graph = s.in_graph || capturing_;
    return s.ptr;
  }
  if (capturing_) {
    void* fresh = owned_count_ < 4 ? zeroed(want, stream_) : nullptr;
    if (fresh != nullptr) owned_[owned_count_++] = fresh;
    return fresh;
  }
  if (s.in_graph && want < 2 * s.bytes) want = 2 * s.bytes;   // what is retired stays below what is in use
  void* fresh = zeroed(want, stream_);
  if (fresh == nullptr) return nullptr;
  if (s.ptr != nullptr) {
    if (s.in_graph) s.retired.push_back(s.ptr);
    else cudaFreeAsync(s.ptr, stream_);
  }
  s.ptr = fresh;
  s.bytes = want;
  s.dirty = s.in_graph = false;
  return fresh;
}

size_t stream_scratch_bytes(cudaStream_t stream, int kind) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  auto it = g_scratch.find(std::make_pair(std::make_pair(dev, stream), kind));
  return it == g_scratch.end() ? 0 : it->second.bytes;
}

void stream_scratch_mark_dirty(int kind) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  for (auto& kv : g_scratch)
    if (kv.first.first.first == dev && kv.first.second == kind) kv.second.dirty = true;
}

void stream_scratch_release(cudaStream_t stream) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  for (auto it = g_scratch.begin(); it != g_scratch.end();) {
    if (it->first.first.first == dev && it->first.first.second == stream) {
      if (it->second.ptr != nullptr) cudaFreeAsync(it->second.ptr, stream);
      for (void* p : it->second.retired) cudaFreeAsync(p, stream);
      it = g_scratch.erase(it);
    } else {
      ++it;
    }
  }
  cudaGetLastError();
}

int cluster_capacity(int s) {
  static std::mutex mu;
  static int known[64][kMaxClusterSplit + 1] = {};   // capacity + 1
  constexpr int kSmem = 200 * 1024;                  // one CTA per SM
  int dev = 0;
  if (s < 2 || s > kMaxClusterSplit || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  int& slot = known[dev][s];
  if (slot == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = kSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = s;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(full_sm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, full_sm_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    slot = n + 1;
  }
  return slot - 1;
}

bool programmatic_launch_enabled() {
  static const bool enabled = std::getenv("KS_B200_NO_PDL") == nullptr;
  return enabled;
}

}  // namespace sm100
}  // namespace ksb
