// Load cases, FP32 vectors.
#include "multi.cuh"
#include "launch.h"

namespace pgi {

const void* multi32_kernel(int cases) {
    return cases == 2 ? (const void*)pg::pcg_multi_kernel<float, true, 2> : (const void*)pg::pcg_multi_kernel<float, true, 4>;
}

}  // namespace pgi
