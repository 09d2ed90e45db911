// Host-side helpers shared by the sm_100a kernels: TMA tensor-map encoding
// through the driver entry point (no link-time dependency on libcuda) and a
// per-(device, stream) scratch allocation for kernels that need workspace.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

namespace ksb {
namespace sm100 {

// True when cuTensorMapEncodeTiled could be resolved.
bool tma_available();

// Encodes a tiled tensor map of rank 2 or 3 (dimension 0 innermost).
// strides_bytes has rank-1 entries (strides of dimensions 1..rank-1, multiples
// of 16 bytes); base must be 16-byte aligned; box[0] * element size must be a
// multiple of 16 bytes and, with a swizzle, at most the swizzle span.
bool tma_encode(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base, const uint64_t* dims,
                const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle);

// Library-owned scratch memory of the current device and one stream, for the host thread that holds
// this object: what it gets and what it enqueues on it before the object goes is one step, with no other
// thread's calls on that stream in between. (Without that another thread's launches could overwrite
// a map between the launch that writes and the one that reads it, or free a buffer by growing it.)
class StreamScratch {
 public:
  explicit StreamScratch(cudaStream_t stream);
  ~StreamScratch();
  StreamScratch(const StreamScratch&) = delete;
  StreamScratch& operator=(const StreamScratch&) = delete;
  // At least `bytes` bytes for one purpose (`kind`: buffers of different kinds never share memory), zero-
  // filled when (re)allocated or marked dirty. Growth is stream-ordered (cudaMallocAsync / cudaFreeAsync),
  // so work already queued on the stream keeps its buffer. NULL when the allocation fails.
  // Under stream capture the stream's buffer serves if it is large enough, and from then on outlives its
  // growth, since a graph holds its address; otherwise the graph gets memory of its own, from here to the
  // end of this object (an allocation and a free node), and nothing is kept. (A buffer first allocated
  // under capture is the graph's: kept for later calls, its address would be used while no graph runs.)
  void* get(size_t bytes, int kind);
  // Under capture, and the stream has no buffer that would serve.
  bool cold_capture(size_t bytes, int kind) const;

 private:
  cudaStream_t stream_;
  int dev_ = -1;
  bool capturing_ = false;
  int owned_count_ = 0;
  void* owned_[4];   // the graph's own memory
  std::unique_lock<std::mutex> lock_;
};
// Size of a stream's buffer (0 when none exists).
size_t stream_scratch_bytes(cudaStream_t stream, int kind);
// Marks every buffer of `kind` on the current device as possibly modified by a kernel
// that stopped half-way: it is cleared before its next use.
void stream_scratch_mark_dirty(int kind);
// Frees (stream-ordered) every buffer of the current device that belongs to `stream`;
// called when the stream is destroyed, so that a recycled handle starts clean.
void stream_scratch_release(cudaStream_t stream);

// Launches `kernel` with programmatic stream serialization: it may begin while the kernel
// before it on the stream is still running, once every CTA of that kernel has executed
// griddepcontrol.launch_dependents or exited (a kernel that never executes it is simply
// waited for, as in an ordinary launch). The launched kernel must order its own accesses
// with griddepcontrol.wait (grid_dependency_wait() in sm100_ptx.cuh).
// False when the environment variable KS_B200_NO_PDL is set (read once): launch_programmatic
// then launches the ordinary way.
bool programmatic_launch_enabled();

template <typename... KArgs, typename... Args>
inline cudaError_t launch_programmatic(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem,
                                       cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = programmatic_launch_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// The same with the grid cut into clusters of `cluster` CTAs (1: no clusters), and the ordinary way unless `programmatic`.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_programmatic_cluster(void (*kernel)(KArgs...), unsigned grid, unsigned cluster, bool programmatic,
                                               unsigned block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (programmatic && programmatic_launch_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Clusters of `s` CTAs (2 <= s <= kMaxClusterSplit) that the current device runs at a time when
// a CTA fills an SM: a cluster's CTAs sit in one group of SMs, so 148 SMs hold fewer than
// 148 / s. 0 when the query fails. Cached per device.
constexpr int kMaxClusterSplit = 8;   // portable cluster size
int cluster_capacity(int s);

}  // namespace sm100
}  // namespace ksb
