// Fakes of the runtime calls that pb_launch.cuh makes on the host: linked into a
// program, they take the place of the shared runtime's.
#include "runtime_fakes.hpp"

namespace fakes {
cudaError_t last = cudaSuccess, launch_result = cudaSuccess, attribute_result = cudaSuccess;
int attribute_calls = 0;
}  // namespace fakes

extern "C" {
cudaError_t cudaGetLastError() {
  const cudaError_t e = fakes::last;
  fakes::last = cudaSuccess;
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
  return fakes::last = fakes::launch_result;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st) {
  *st = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* dev) {
  *dev = 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  ++fakes::attribute_calls;
  return fakes::last = fakes::attribute_result;
}
}
