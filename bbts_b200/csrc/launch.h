// Launch of a kernel that may start before its predecessor in the stream has
// finished (programmatic dependent launch): the kernel runs griddep_wait (ptx.cuh)
// before it touches memory. Its launch latency and prologue then overlap the
// predecessor's tail. Behind anything but such a kernel it is a plain launch. The f32
// SIMT products and the quantisation kernels have no such wait and launch plainly.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace bbx {

// While one lives (with on = true), its thread's launches are plain: a kernel
// that starts early holds its shared memory while it waits, which costs a kernel of
// another stream that could run there meanwhile. The executors use it where
// streams overlap (an uneven DAG's gathers kept its matmuls off the SMs: 1593 -> 1635 us).
class PlainLaunches {
 public:
  explicit PlainLaunches(bool on) : before_(active()) { active() = before_ || on; }
  ~PlainLaunches() { active() = before_; }
  PlainLaunches(const PlainLaunches&) = delete;
  PlainLaunches& operator=(const PlainLaunches&) = delete;
  static bool& active() {
    static thread_local bool on = false;
    return on;
  }

 private:
  bool before_;
};

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = PlainLaunches::active() ? 0 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
}

}  // namespace bbx
