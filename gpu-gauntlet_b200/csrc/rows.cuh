// The operator as assembled 3x3 node blocks ("row blocks"), the form the
// persistent PCG kernels multiply with.
//
// Row n of a part holds one slot per node m that shares an element with n
// (n itself included): the block K_nm = sum of the shared elements' 3x3
// blocks, added in FP64 in element order and rounded once for FP32 solves.
// Slots are sorted by global node id, so the parts that hold a row (its
// owner, and with a 2-ring halo its neighbours) have the same slots in the
// same order and compute the same bits.
//
// Rows are taken in groups of 10, one warp a group: lanes 3 i, 3 i + 1 and
// 3 i + 2 share row i of the group and take its slots in turn (lane 3 i + d
// slots d, d + 3, ...), each adding its slots' blocks to all three
// components; two shuffles then give lane 3 i + d component d.  A group is
// stored as q-steps (slots 3 q .. 3 q + 2 of its rows): 30 columns and
// 9 x 30 block entries (row-major 3 r + c, then lane), so consecutive lanes
// read consecutive words; rows with fewer slots are padded with zero blocks.
//
// Why: an assembled row of the Q4 grid has 9 blocks (648 B in FP64), its
// four element tasks 4 x 36 entries (1,152 B) whose results had to be
// written and gathered again behind a barrier.  K u was bound by the
// shared-memory reads of those entries.  A warp's first group stays in
// registers (3 q-steps: 27 entries a lane), so the parts of the
// 60k-DOF plate read no coefficients at all; a lane reads u of a slot's node
// once for three components (9 loads a lane where a thread per component
// needs 27).
//
// FP32 rows of Q4 plates multiply w's difference to the row's own node.  A
// translation in w has no stiffness there (sum_m K_nm e_w = 0: the shape
// functions' gradients sum to zero), so for a smooth u the products with w are
// large and cancel: rounded to FP32 their sum had 1.6 times the error of the
// element form (lowest mode of a clamped 141 x 141 plate: 7.4e-2 of |K u|), and
// mixed solves that converged with the element form stagnated.
// sum_m K_nm (w_m - w_n, thx_m, thy_m) is the same sum, its differences are
// almost exact, and its error there is 1.0e-3.  Cost, a load and three
// subtractions a lane, at equal iterations on the 60k-DOF plate (ms on the
// device): block Jacobi 4.64 -> 4.73, with the smoother 3.28 -> 3.43, two-level
// Chebyshev 1.26 -> 1.30.  It returns elsewhere: of the 256-plate batch in mixed
// precision 44 plates stagnated (element form 71), now 3 to 5.  FP64 rows keep the plain form, FP64 has the
// digits; so do DKT rows: the reference's element, which this one restates, does
// have stiffness in a translation (and few iterations).
#pragma once

#include <cstdint>

namespace pg {

constexpr int kRowGroup = 10;   // rows per group (3 lanes each: 30 of a warp's 32)
constexpr int kRowLanes = 30;
constexpr int kRegSteps = 3;    // q-steps of a resident group kept in registers

// s += the blocks k[9 (q - qa) ..][lane] of q-steps [qa, qb) times u at the
// columns c[q - qa][lane], its w less w0 (0, or the row's own w; FP32 only).
template <typename T>
__device__ __forceinline__ void row_steps(const T* __restrict__ u, const uint16_t* __restrict__ c,
                                          const T* __restrict__ k, int steps, T w0, T (&s)[3]) {
#pragma unroll 3
    for (int q = 0; q < steps; q++) {
        const T* v = u + 3 * (int)c[q * kRowLanes];
        const T v0 = sizeof(T) == 4 ? v[0] - w0 : v[0], v1 = v[1], v2 = v[2];
        const T* b = k + q * 9 * kRowLanes;
#pragma unroll
        for (int r = 0; r < 3; r++)
            s[r] = fma(b[(3 * r + 2) * kRowLanes], v2,
                       fma(b[(3 * r + 1) * kRowLanes], v1, fma(b[3 * r * kRowLanes], v0, s[r])));
    }
}

// Lane 3 i + d holds its share s of row i's three components: the sum of
// component d over the row's three lanes, in an order that depends on d
// alone.  Every lane of the warp calls it.
template <typename T>
__device__ __forceinline__ T row_join(const T (&s)[3]) {
    const int lane = threadIdx.x & 31, d = lane % 3, b = lane - d;
    // lane d sends component d + 1 to lane d + 1 and component d + 2 to lane d + 2
    const T up = d == 0 ? s[1] : d == 1 ? s[2] : s[0];
    const T dn = d == 0 ? s[2] : d == 1 ? s[0] : s[1];
    const T own = d == 0 ? s[0] : d == 1 ? s[1] : s[2];
    const T f1 = __shfl_sync(0xffffffffu, up, b + (d + 2) % 3);
    const T f2 = __shfl_sync(0xffffffffu, dn, b + (d + 1) % 3);
    return own + f1 + f2;
}

// Component d of D_n^-1 v for the node of lanes 3 i .. 3 i + 2, lane 3 i + d
// holding v_d and row d of the node's 3x3 inverse from column d on, cyclically
// (b[0] = B_dd, b[1] = B_d,d+1, b[2] = B_d,d+2).  All lanes of the warp call it.
template <typename T>
__device__ __forceinline__ T jacobi_lane(const T (&b)[3], T v) {
    const int lane = threadIdx.x & 31, d = lane % 3, l0 = lane - d;
    const T v1 = __shfl_sync(0xffffffffu, v, l0 + (d + 1) % 3);
    const T v2 = __shfl_sync(0xffffffffu, v, l0 + (d + 2) % 3);
    return b[0] * v + b[1] * v1 + b[2] * v2;
}

}  // namespace pg
