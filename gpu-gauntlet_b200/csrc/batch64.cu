// Batches, FP64.
#include "kernels.cuh"
#include "launch.h"

namespace pgi {

const void* batch64_kernel(bool coarse, bool cheb) {
    if (coarse)
        return cheb ? (const void*)pg::pcg_batch_kernel<double, false, true, true> : (const void*)pg::pcg_batch_kernel<double, false, true, false>;
    return cheb ? (const void*)pg::pcg_batch_kernel<double, false, false, true> : (const void*)pg::pcg_batch_kernel<double, false, false, false>;
}

}  // namespace pgi
