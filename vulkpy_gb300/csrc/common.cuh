// Internal definitions shared by the runtime and the kernel files.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>
#include <cstdio>
#include <cstdarg>
#include <atomic>
#include <mutex>
#include <string>
#include <utility>
#include <unordered_map>
#include <vector>

#include "../../include/vulkpy_gb300.h"

#define VKC_EXPORT extern "C" __attribute__((visibility("default")))

namespace vkc {
// Whether this thread's calls go to a branch of a device (BranchScope,
// vkc_side_begin) and whether it defers the joins (vkc_side_defer).
struct ThreadBranch {
  const void* of = nullptr;        // the device's CurrentStream
  cudaStream_t stream = nullptr;
  const void* deferred = nullptr;  // the device whose joins wait
};
inline thread_local ThreadBranch t_branch;

// The stream that calls on a device go to: the shared one (the device's own
// or the user's), or while this thread works on a branch, the branch's.  A
// branch is the thread's and not the device's: the interpreter runs other
// threads in the middle of a training step, and what they queue must not
// land on the step's branch, which their later calls are not ordered after.
struct CurrentStream {
  cudaStream_t shared = nullptr;
  operator cudaStream_t() const { return t_branch.of == this ? t_branch.stream : shared; }
};

class BranchScope {
 public:
  BranchScope(const CurrentStream& current, cudaStream_t stream) : before_(t_branch) {
    t_branch.of = &current;
    t_branch.stream = stream;
  }
  ~BranchScope() {
    t_branch.of = before_.of;
    t_branch.stream = before_.stream;
  }
  BranchScope(const BranchScope&) = delete;
  BranchScope& operator=(const BranchScope&) = delete;

 private:
  ThreadBranch before_;
};
}  // namespace vkc

struct vkc_device {
  int index = 0;
  int sm_count = 0;
  int cc_major = 0, cc_minor = 0;
  cudaStream_t own_stream = nullptr;   // compute stream created at open
  vkc::CurrentStream stream;           // current compute stream (own, user's or this thread's branch)
  cudaStream_t copy_stream = nullptr;  // uploads into fresh buffers
  cudaMemPool_t upload_pool = nullptr; // their buffers (reused only by later uploads)
  // Upload buffers the caller freed, each with an event on the compute stream
  // after its last use: the next upload of the same size takes one (waiting
  // on that event if needed) instead of allocating (vkc_free / vkc_upload*).
  struct UploadBlock {
    void* ptr;
    size_t bytes;
    cudaEvent_t freed;
  };
  std::vector<UploadBlock> upload_free;
  std::unordered_map<void*, size_t> upload_live;  // upload buffers in use, by size
  cudaEvent_t copy_done = nullptr;     // reused marker for uploads
  cudaStream_t d2h_stream = nullptr;   // asynchronous read-backs (vkc_d2h_async)
  cudaEvent_t d2h_after = nullptr;     // reused marker: compute work a read-back follows
  cudaStream_t side_stream = nullptr;  // independent work forked from `stream` inside one call
  cudaStream_t bias_stream = nullptr;  // a second such branch (the Dense backward's bias sums)
  cudaEvent_t side_fork = nullptr, side_join = nullptr, bias_join = nullptr;
  std::atomic<int> side_pending{0};    // branches forked and not yet joined back
  uint32_t* err_word = nullptr;        // device error flags (bit0: gather index)
  uint32_t* done_ctr = nullptr;        // arrival counter of last-block reductions (zero between kernels)
  uint32_t* xo_jump_pows = nullptr;    // xoshiro jump-map powers (lazy)
  uint32_t* xo_next_pows = nullptr;    // xoshiro next-map powers (lazy)
  std::mutex mu;
  char name[256] = {0};
};

struct vkc_job {
  cudaEvent_t ev = nullptr;
  int device = 0;
};

namespace vkc {

// Record an error message for vkc_last_error() and return `code`.
int set_error(int code, const char* fmt, ...);
void clear_error();

// Make `dev` current on this thread; returns VKC_OK or an error code.
int bind(vkc_device_t dev);

extern std::atomic<uint64_t> g_launches;  // kernels launched (all devices)

// Counts an allocation request and reports whether an injected failure
// (vkc_inject_alloc_failure) falls on it.
bool alloc_should_fail();

inline int check_launch(const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(VKC_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
  return VKC_OK;
}

// Grid for a grid-stride streaming kernel with `threads` per block.
inline unsigned stream_grid(const vkc_device* dev, size_t work_items, int threads, int blocks_per_sm = 8) {
  size_t want = (work_items + threads - 1) / threads;
  size_t cap = (size_t)dev->sm_count * blocks_per_sm;
  if (want < 1) want = 1;
  return (unsigned)(want < cap ? want : cap);
}

// Blocks of `kernel` resident per SM at `threads` threads and `smem` bytes of
// dynamic shared memory (cudaOccupancyMaxActiveBlocksPerMultiprocessor,
// cached per kernel; at least 1).
int resident_blocks(const void* kernel, int threads, size_t smem = 0);

// Grid for a grid-stride kernel: at most one full wave of resident blocks.
// A grid sized for more blocks than fit (e.g. 8 per SM for a kernel whose
// registers allow 5) runs a partial second wave that leaves SMs idle at the
// end of the launch.
template <class K>
inline unsigned wave_grid(const vkc_device* dev, K* kernel, size_t work_items, int threads, size_t smem = 0) {
  size_t want = (work_items + threads - 1) / threads;
  if (want < 1) want = 1;
  const size_t cap = (size_t)dev->sm_count * (size_t)resident_blocks((const void*)kernel, threads, smem);
  return (unsigned)(want < cap ? want : cap);
}

// Loads kernels on the device (once; `done` has a bit per device).  A kernel is
// otherwise loaded at its first launch, and the host then waits for the work
// running before it: a call of several launches loads all of them first, so
// that its first run is asynchronous too.
template <class... K>
inline void load_kernels(vkc_device_t dev, std::atomic<uint64_t>& done, K*... kernels) {
  const uint64_t bit = uint64_t(1) << (dev->index & 63);
  if (done.load(std::memory_order_acquire) & bit) return;
  cudaFuncAttributes at;
  const bool ok = ((cudaFuncGetAttributes(&at, (const void*)kernels) == cudaSuccess) && ...);
  if (!ok) {
    cudaGetLastError();  // the launch will say what is wrong
    return;
  }
  done.fetch_or(bit, std::memory_order_release);
}

// Stream-ordered scratch allocation on the device's current stream.
int scratch_alloc(vkc_device_t dev, size_t bytes, void** p);
void scratch_free(vkc_device_t dev, void* p);

// scratch_alloc for scratch that the call can do without.  While the stream is
// captured an allocation that does not fit fails only when the graph is
// launched, so from 256 MiB on it is refused there unless the device has twice
// as much free.
int scratch_alloc_optional(vkc_device_t dev, size_t bytes, void** p);

// ---- programmatic dependent launch (PDL)
// A kernel launched with launch_pdl may be scheduled while the kernel before
// it on the stream is still running: its blocks become resident as that
// kernel's blocks trigger (pdl_trigger) or exit, then wait in pdl_wait()
// until it has completed and its memory is visible.  So the launch gap and
// the block scheduling of consecutive short kernels overlap.  Every kernel
// launched this way calls pdl_wait() before it touches global memory (after
// it, everything the previous kernel wrote is visible, as after an ordinary
// launch); without the launch attribute both calls are no-ops.
extern std::atomic<int> g_pdl;             // 1: launch_pdl adds the attribute (vkc_set_pdl)
extern std::atomic<int> g_cluster_splitk;  // 1: split-K reduced inside the GEMM (vkc_set_cluster_splitk)

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_pdl.load(std::memory_order_relaxed) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// The second kernel of a two-kernel op over n elements: with PDL from 2^21 on,
// where the GPU is the bound and its launch then overlaps the first kernel's
// tail (7 reductions over 60 x 8192 x 9: 272 -> 253 us); below, the calls are
// bound by the host, and the plain launch costs it less (133 -> 130 us for 13
// calls on 100 x 100).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_second(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, size_t n,
                                 Args&&... args) {
  if (n >= (size_t(1) << 21)) return launch_pdl(kern, grid, block, 0, stream, std::forward<Args>(args)...);
  kern<<<grid, block, 0, stream>>>(std::forward<Args>(args)...);
  return cudaSuccess;  // check_launch reads the launch's error
}

// launch_pdl with the blocks grouped into 1-D thread-block clusters of
// `cluster` CTAs (grid.x a multiple of it).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      unsigned cluster, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_pdl.load(std::memory_order_relaxed) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace vkc

#define VKC_CUDA(call)                                                                   \
  do {                                                                                   \
    cudaError_t e__ = (call);                                                            \
    if (e__ != cudaSuccess)                                                              \
      return vkc::set_error(VKC_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e__));     \
  } while (0)

#define VKC_REQUIRE(cond, ...)                                                           \
  do {                                                                                   \
    if (!(cond)) return vkc::set_error(VKC_ERR_INVALID, __VA_ARGS__);                    \
  } while (0)

#define VKC_BIND(dev)                                                                    \
  do {                                                                                   \
    int r__ = vkc::bind(dev);                                                            \
    if (r__ != VKC_OK) return r__;                                                       \
  } while (0)
