// Load cases, FP64.
#include "multi.cuh"
#include "launch.h"

namespace pgi {

const void* multi64_kernel(int cases) {
    return cases == 2 ? (const void*)pg::pcg_multi_kernel<double, false, 2> : (const void*)pg::pcg_multi_kernel<double, false, 4>;
}

}  // namespace pgi
