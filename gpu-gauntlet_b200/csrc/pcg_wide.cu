// One plate with more than kLeanThreads threads a block.
#include "kernels.cuh"
#include "launch.h"

namespace pgi {

namespace {

template <typename T, bool MIXED>
const void* of(bool coarse, bool cheb) {
    if (coarse)
        return cheb ? (const void*)pg::pcg_kernel<T, MIXED, pg::kMaxThreads, true, true> : (const void*)pg::pcg_kernel<T, MIXED, pg::kMaxThreads, true, false>;
    return cheb ? (const void*)pg::pcg_kernel<T, MIXED, pg::kMaxThreads, false, true> : (const void*)pg::pcg_kernel<T, MIXED, pg::kMaxThreads, false, false>;
}

}  // namespace

const void* pcg_wide_kernel(bool mixed, bool coarse, bool cheb) {
    return mixed ? of<float, true>(coarse, cheb) : of<double, false>(coarse, cheb);
}

}  // namespace pgi
