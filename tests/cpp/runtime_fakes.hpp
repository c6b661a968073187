#pragma once

#include <cuda_runtime_api.h>

namespace fakes {
extern cudaError_t last, launch_result, attribute_result;
extern int attribute_calls;
}  // namespace fakes
