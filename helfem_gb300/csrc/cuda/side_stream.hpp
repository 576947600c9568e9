// A second stream for a stage that runs beside another one.
#pragma once

#include <cuda_runtime.h>

namespace hfg {
// a second stream with a fork and a join event (owned by the caller)
struct SideStream {
  cudaStream_t s = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
}  // namespace hfg
