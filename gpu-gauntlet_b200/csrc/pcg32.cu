// One plate, FP32 vectors.
#include "kernels.cuh"
#include "launch.h"

namespace pgi {

const void* pcg32_kernel(bool coarse, bool cheb) {
    if (coarse)
        return cheb ? (const void*)pg::pcg_kernel<float, true, pg::kLeanThreads, true, true> : (const void*)pg::pcg_kernel<float, true, pg::kLeanThreads, true, false>;
    return cheb ? (const void*)pg::pcg_kernel<float, true, pg::kLeanThreads, false, true> : (const void*)pg::pcg_kernel<float, true, pg::kLeanThreads, false, false>;
}

}  // namespace pgi
