// Host side of pb_launch.cuh on fakes of the runtime calls: no GPU is touched.
#include <cstdio>

#include "pb_launch.cuh"
#include "runtime_fakes.hpp"

struct Args {
  int x;
};
__global__ void kernel(const Args) {}

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok) {
    std::printf("failed: %s\n", what);
    ++failures;
  }
}

int main() {
  // a refused launch or attribute is returned and not left for the next caller
  fakes::launch_result = cudaErrorInvalidConfiguration;
  check(pb::pb_launch<Args>(kernel, 1, 4096, 0, nullptr, Args{0}) == cudaErrorInvalidConfiguration, "launch error");
  check(cudaGetLastError() == cudaSuccess, "launch error left behind");
  fakes::attribute_result = cudaErrorInvalidValue;
  check(pb::pb_allow_smem<kernel>(1 << 30) == cudaErrorInvalidValue, "attribute error");
  check(cudaGetLastError() == cudaSuccess, "attribute error left behind");
  if (failures == 0) std::printf("launch ok\n");
  return failures;
}
