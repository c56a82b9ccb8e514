// The run-time-plan row passes and the 1D passes, FP32 (passes.cuh, long1d.cuh).
#define CSIPM_PASSES_HERE
#include "long1d.cuh"

namespace csipm {

#define CSIPM_X(...) CSIPM_PASS_R(, __VA_ARGS__)
CSIPM_ROW_LIST32(CSIPM_X)
#undef CSIPM_X
#define CSIPM_X(...) CSIPM_PASS_1D(, __VA_ARGS__)
CSIPM_1D_LIST32(CSIPM_X)
#undef CSIPM_X

}  // namespace csipm
