// One plate, FP64.
#include "kernels.cuh"
#include "launch.h"

namespace pgi {

const void* pcg64_kernel(bool coarse, bool cheb) {
    if (coarse)
        return cheb ? (const void*)pg::pcg_kernel<double, false, pg::kLeanThreads, true, true> : (const void*)pg::pcg_kernel<double, false, pg::kLeanThreads, true, false>;
    return cheb ? (const void*)pg::pcg_kernel<double, false, pg::kLeanThreads, false, true> : (const void*)pg::pcg_kernel<double, false, pg::kLeanThreads, false, false>;
}

}  // namespace pgi
