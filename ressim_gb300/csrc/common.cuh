// Shared infrastructure of the resgpu library: context, device buffers,
// launch accounting, error propagation across the C ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <map>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/rsg.h"
#include "perdevice.hpp"

namespace rsg {

// Thrown inside the library, converted to an rsg_status at the C boundary.
struct Error : std::runtime_error {
  rsg_status status;
  Error(rsg_status s, const std::string& m) : std::runtime_error(m), status(s) {}
};

#define RSG_CUDA(call)                                                                         \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess)                                                                     \
      throw ::rsg::Error(RSG_CUDA_ERROR, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

template <class T>
struct DeviceBuffer {
  T* ptr = nullptr;
  size_t count = 0;
  DeviceBuffer() {}
  explicit DeviceBuffer(size_t n) { resize(n); }
  DeviceBuffer(const DeviceBuffer&) = delete;
  DeviceBuffer& operator=(const DeviceBuffer&) = delete;
  DeviceBuffer(DeviceBuffer&& o) noexcept : ptr(o.ptr), count(o.count) {
    o.ptr = nullptr;
    o.count = 0;
  }
  DeviceBuffer& operator=(DeviceBuffer&& o) noexcept {
    release();
    ptr = o.ptr;
    count = o.count;
    o.ptr = nullptr;
    o.count = 0;
    return *this;
  }
  ~DeviceBuffer() { release(); }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    count = 0;
  }
  void resize(size_t n) {
    if (n == count && ptr) return;
    release();
    if (n) RSG_CUDA(cudaMalloc(&ptr, n * sizeof(T)));
    count = n;
  }
  T* get() const { return ptr; }
  size_t size() const { return count; }
};

struct ProfileEntry {
  double ms = 0;
  int64_t launches = 0;
};

struct Context {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  int cluster_size = 8;  // CTAs per cluster of the level-scheduled sweeps
  int64_t launches = 0;
  std::string last_error;
  bool profiling = false;
  struct Pending {
    std::string name;
    cudaEvent_t a, b;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> event_pool;
  std::map<std::string, ProfileEntry> profile;
  // pinned host staging for small scalar reads
  void* pinned = nullptr;
  cudaEvent_t timers[64] = {};
  // set by kernels whose bounded waits ran out (1 + site); read after solves
  DeviceBuffer<int> dev_err;

  void open();   // stream, staging page, error flag; device and num_sms are set
  void close();  // gives them back
  // Takes over what another context, standing in for this one, has counted.
  void take_counts(Context& other);

  cudaEvent_t get_event();
  void flush_profile();  // requires a synchronized stream
  void sync();
  // throws RSG_TIMEOUT (and clears the flag) when a kernel's bounded wait ran out
  void check_device_error();
};

// Launch helper: counts launches and (optionally) brackets them with events.
struct LaunchScope {
  Context& ctx;
  const char* name;
  cudaEvent_t a = nullptr;
  LaunchScope(Context& c, const char* n) : ctx(c), name(n) {
    ctx.launches++;
    if (ctx.profiling) {
      a = ctx.get_event();
      cudaEventRecord(a, ctx.stream);
    }
  }
  ~LaunchScope() {
    if (ctx.profiling) {
      cudaEvent_t b = ctx.get_event();
      cudaEventRecord(b, ctx.stream);
      ctx.pending.push_back({name, a, b});
    }
  }
};

inline void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw Error(RSG_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
}

// an empty grid (nothing to do, e.g. a mesh without connections) launches nothing
inline bool grid_empty(int g) { return g <= 0; }
inline bool grid_empty(const dim3& g) { return g.x == 0 || g.y == 0 || g.z == 0; }

#define RSG_LAUNCH(ctx, name, kernel, grid, block, smem, ...)                    \
  do {                                                                           \
    if (::rsg::grid_empty(grid)) break;                                          \
    ::rsg::LaunchScope scope_(ctx, name);                                        \
    kernel<<<(grid), (block), (smem), (ctx).stream>>>(__VA_ARGS__);              \
    ::rsg::check_launch(name);                                                   \
  } while (0)

// Launch of a kernel that begins with chain_begin() or chain_wait(): its blocks
// may start while the last ones of the kernel before it in the stream still run,
// and wait there (programmatic dependent launch).  An iteration of a Krylov
// solver is a chain of 9 to 11 kernels, each idle for about 2 us at its start and
// end on small systems: chained, a 32x32x8 two-phase step takes 8% less, the 64x64
// potential problem 11%, the 128x128x32 mixed solve 8%.
template <typename... P, typename... A>
inline void launch_chained(Context& ctx, const char* name, void (*kernel)(P...), int grid, int block, size_t smem,
                           A&&... args) {
  if (grid <= 0) return;
  LaunchScope scope(ctx, name);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) throw Error(RSG_CUDA_ERROR, std::string(name) + ": " + cudaGetErrorString(e));
}

#ifdef __CUDACC__
// Before a chained kernel's first access to global memory: waits for the
// kernel before it to end (everything it wrote is then visible).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel's blocks start, as far as there is room beside this
// one's, once every block has come here or ended.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;"); }
// Both at once, for kernels of few blocks or of one a SM, beside which the next
// kernel's blocks spread over the SMs, and for the V-cycle's, whose next kernel
// is mostly a sweep of one CTA.  Others call chain_next() late (krylov.cu).
__device__ __forceinline__ void chain_begin() {
  chain_wait();
  chain_next();
}
#endif

// Lets `kernel` use `bytes` of dynamic shared memory on the context's device;
// done: the kernel's own (static) record of where it may.
template <typename Kernel>
inline void allow_smem(PerDevice& done, const Context& ctx, Kernel kernel, size_t bytes) {
  done.ask(ctx.device, [&] {
    RSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return true;
  });
}

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

// Runs f and converts exceptions to a status, recording the message.
template <class F>
rsg_status guarded(Context* ctx, F&& f) {
  try {
    f();
    return RSG_OK;
  } catch (const Error& e) {
    if (ctx) ctx->last_error = e.what();
    return e.status;
  } catch (const std::bad_alloc&) {
    if (ctx) ctx->last_error = "host allocation failed";
    return RSG_CUDA_ERROR;
  } catch (const std::exception& e) {
    if (ctx) ctx->last_error = e.what();
    return RSG_BAD_ARG;
  }
}

}  // namespace rsg

struct rsg_ctx {
  rsg::Context c;
};
