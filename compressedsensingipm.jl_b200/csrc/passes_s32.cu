// The run-time-plan strided passes, FP32 (passes.cuh).
#define CSIPM_PASSES_HERE
#include "passes.cuh"

namespace csipm {

#define CSIPM_X(...) CSIPM_PASS_S(, __VA_ARGS__)
CSIPM_STRIDED_LIST32(CSIPM_X)
#undef CSIPM_X

}  // namespace csipm
