// Launches of the pass kernels that overlap the end of the kernel before them
// in the stream (programmatic dependent launch).
//
// The passes of a transform follow one another on one stream.  A pass kernel
// starts while its predecessor's last CTAs still run, reads what no kernel
// writes (tile descriptors, piece rows, twiddles: the plan's tables) and waits
// with pb_dependency_wait before its first read of the data and, being before
// that, before any write.  Each kernel lets its successor start when its own
// last tiles begin.  A wait ends when every earlier kernel of the stream has
// completed and its writes are visible.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace pb {

// Waits for the preceding kernels of the stream (no effect in a kernel
// launched without the attribute).  src0 and src1 are the offsets that the
// first two tiles' reads of the data are computed from: passing them through
// the wait keeps those reads behind it.
__device__ __forceinline__ void pb_dependency_wait(long long& src0, long long& src1) {
  asm volatile("griddepcontrol.wait;" : "+l"(src0), "+l"(src1)::"memory");
}
__device__ __forceinline__ void pb_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pb_allow_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether a gated pass has been rejected (every thread; waits for the check).
__device__ __forceinline__ bool pb_rejected(const int* gate) {
  if (gate == nullptr) return false;
  pb_dependency_wait();
  return *reinterpret_cast<const volatile int*>(gate) != 0;
}

// An error that the caller returns, taken off the runtime's record: left there,
// the next call that ends in cudaGetLastError (a launch with <<<>>>, the host
// program's own check) would report it for work that was fine.
inline cudaError_t pb_reported(cudaError_t err) {
  if (err != cudaSuccess) (void)cudaGetLastError();
  return err;
}

// cudaFuncAttributeMaxDynamicSharedMemorySize of KERN, set once per device.
template <auto KERN>
inline cudaError_t pb_allow_smem(int bytes) {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (bit != 0 && (done.load(std::memory_order_relaxed) & bit)) return cudaSuccess;
  err = pb_reported(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  if (err == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return err;
}

// Launches `kern` overlapped.  In a stream capture the launch is a plain one:
// the graph keeps full dependencies between its nodes.
template <typename Args>
inline cudaError_t pb_launch(void (*kern)(const Args), long long grid, int threads, size_t smem, cudaStream_t stream,
                             const Args& args) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  const bool known = cudaStreamIsCapturing(stream, &capturing) == cudaSuccess;
  if (!known) (void)cudaGetLastError();
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = known && capturing == cudaStreamCaptureStatusNone ? 1 : 0;
  return pb_reported(cudaLaunchKernelEx(&cfg, kern, args));
}

}  // namespace pb
