// Batches, FP32 vectors.
#include "kernels.cuh"
#include "launch.h"

namespace pgi {

const void* batch32_kernel(bool coarse, bool cheb) {
    if (coarse)
        return cheb ? (const void*)pg::pcg_batch_kernel<float, true, true, true> : (const void*)pg::pcg_batch_kernel<float, true, true, false>;
    return cheb ? (const void*)pg::pcg_batch_kernel<float, true, false, true> : (const void*)pg::pcg_batch_kernel<float, true, false, false>;
}

}  // namespace pgi
