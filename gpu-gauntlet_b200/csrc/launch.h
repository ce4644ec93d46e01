// The persistent kernels' entry points, by method.  Each file that defines some of
// them is a device module of its own, which the driver loads when one of its
// kernels is first used.  In one module with the set-up kernels, the first call of a
// process loaded all 28 instantiations: 27 ms for a 44k-DOF triangle plate with block
// Jacobi, 31 for the 60k-DOF plate with the mixed two-level method; now 8 and 13.
#pragma once

namespace pgi {

const void* pcg64_kernel(bool coarse, bool cheb);              // FP64, up to kLeanThreads
const void* pcg32_kernel(bool coarse, bool cheb);              // FP32 vectors, up to kLeanThreads
const void* pcg_wide_kernel(bool mixed, bool coarse, bool cheb);  // up to kMaxThreads
const void* batch64_kernel(bool coarse, bool cheb);
const void* batch32_kernel(bool coarse, bool cheb);
const void* multi64_kernel(int cases);
const void* multi32_kernel(int cases);

}  // namespace pgi
