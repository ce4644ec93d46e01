// Device set-up of the two-level preconditioner's coarse space:
//   coarse_assemble_kernel  A_c = P^T K P from the FP64 element matrices,
//                           one thread per element, FP64 atomics into A_c
//   coarse_step_kernel      A_c^-1 by blocked Gauss-Jordan elimination, 32
//                           modes a launch, numerically dependent modes
//                           dropped (pivot <= 1e-13 max diagonal)
//   coarse_rows_kernel      each part's rows of A_c^-1 (FP64 and FP32)
// P holds one aggregate per part with the plate's three rigid-body modes
// (w = 1; w = dy, theta_x = 1/h; w = dx, theta_y = -1/h about the
// aggregate centre, h its size), zero on constrained DOFs.
#pragma once

#include <cstdint>

namespace pg {

template <int NPE>
__global__ void coarse_assemble_kernel(int Ne, int C, const float* __restrict__ nodes,
                                       const uint32_t* __restrict__ elements, const uint8_t* __restrict__ cons,
                                       const int* __restrict__ owner, const double* __restrict__ geom,
                                       const double* __restrict__ ke64, double* __restrict__ Ac) {
    constexpr int ND = 3 * NPE;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= Ne) return;
    const double* K = ke64 + (size_t)e * ND * ND;
    double Ph[NPE][3][3];
    int ag[NPE];
    for (int i = 0; i < NPE; i++) {
        const int n = (int)elements[(size_t)e * NPE + i];
        const int a = owner[n];
        ag[i] = a;
        const double ih = geom[3 * a + 2];
        const double dx = ((double)nodes[2 * n] - geom[3 * a]) * ih;
        const double dy = ((double)nodes[2 * n + 1] - geom[3 * a + 1]) * ih;
        const double v[3][3] = {{1.0, dy, dx}, {0.0, ih, 0.0}, {0.0, 0.0, -ih}};
        for (int d = 0; d < 3; d++)
            for (int m = 0; m < 3; m++) Ph[i][d][m] = cons[3 * n + d] ? 0.0 : v[d][m];
    }
    for (int i = 0; i < NPE; i++)
        for (int j = 0; j < NPE; j++) {
            double T[3][3];  // K_ij Phi_j
            for (int d = 0; d < 3; d++)
                for (int m = 0; m < 3; m++) {
                    double acc = 0.0;
                    for (int f = 0; f < 3; f++) acc += K[(3 * i + d) * ND + 3 * j + f] * Ph[j][f][m];
                    T[d][m] = acc;
                }
            for (int mi = 0; mi < 3; mi++)
                for (int mj = 0; mj < 3; mj++) {
                    double acc = 0.0;
                    for (int d = 0; d < 3; d++) acc += Ph[i][d][mi] * T[d][mj];
                    if (acc != 0.0) atomicAdd(Ac + (size_t)(3 * ag[i] + mi) * C + 3 * ag[j] + mj, acc);
                }
        }
}

// *out = the largest diagonal entry of A ([C][C]).  One block.
__global__ void coarse_dmax_kernel(int C, const double* __restrict__ A, double* out) {
    __shared__ double red[32];
    double m = 0.0;
    for (int i = threadIdx.x; i < C; i += blockDim.x) m = fmax(m, A[(size_t)i * C + i]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) m = fmax(m, red[w]);
        *out = m;
    }
}

constexpr int kCoarseTile = 32;      // modes eliminated per step, and the tile of one block
constexpr int kCoarseThreads = 256;  // row tid / 8 of a tile, columns 4 (tid % 8) ..

// One step of the blocked Gauss-Jordan inversion of the SPD matrix A: the
// modes J = [p0, p0 + 32) are eliminated, A -> out ([C][C] each):
//   B = A_JJ^-1, out_JJ = B, out_JK = B A_JK, out_IJ = -A_IJ B,
//   out_IK = A_IK - A_IJ B A_JK
// so A_c^-1 stands in the last step's output after ceil(C / 32) steps.  One
// block per 32 x 32 tile of the matrix; every block inverts the pivot tile by
// itself (32 in-place pivots) and reads only the step's input, so a step is
// one launch with no wait between blocks.  A mode whose pivot is <= 1e-13
// *dmax depends on the others: it is dropped (its row and column of B, and so
// of the inverse, are zero) and counted in *dropped.
// Bound by the 32 dependent pivots of a step (about 3 us) and the launches;
// C = 444 (14 steps): 0.12 ms, where the factorisation in one block with
// inversion of L and L^-T L^-1 took 2.74 ms.
__global__ void __launch_bounds__(kCoarseThreads) coarse_step_kernel(int C, int p0, const double* __restrict__ A,
                                                                     double* __restrict__ out,
                                                                     const double* __restrict__ dmax, int* dropped) {
    constexpr int W = kCoarseTile;
    __shared__ double Bs[W][W + 2], X[W][W + 2], T[W][W + 2];
    __shared__ double rowk[2][W], colk[2][W];
    const int tid = threadIdx.x, i = tid >> 3, j0 = (tid & 7) * 4;
    const int I0 = blockIdx.y * W, K0 = blockIdx.x * W, w = min(W, C - p0);
    const double tol = 1e-13 * *dmax;
    // padding past C: the identity, so its pivots are inert
    auto at = [&](int r0, int c0, int r, int c) -> double {
        return r0 + r < C && c0 + c < C ? A[(size_t)(r0 + r) * C + c0 + c] : 0.0;
    };
    double m[4];
#pragma unroll
    for (int q = 0; q < 4; q++) m[q] = i < w && j0 + q < w ? at(p0, p0, i, j0 + q) : (i == j0 + q ? 1.0 : 0.0);
    unsigned drop = 0;  // the same in every thread
    for (int k = 0; k < W; k++) {
        double* rk = rowk[k & 1];
        double* ck = colk[k & 1];
        if (i == k)
#pragma unroll
            for (int q = 0; q < 4; q++) rk[j0 + q] = m[q];
        if ((k & ~3) == j0) ck[i] = (k & 3) == 0 ? m[0] : (k & 3) == 1 ? m[1] : (k & 3) == 2 ? m[2] : m[3];
        __syncthreads();  // the buffers alternate: the last pivot's may still be read
        const double d = rk[k];
        if (k < w && !(d > tol)) {
            drop |= 1u << k;
            continue;
        }
        const double inv = 1.0 / d, f = ck[i] * inv;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int j = j0 + q;
            if (i == k) m[q] = j == k ? inv : m[q] * inv;
            else m[q] = j == k ? -f : m[q] - f * rk[j];
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const bool kept = !((drop >> i) & 1u) && !((drop >> (j0 + q)) & 1u);
        Bs[i][j0 + q] = kept ? m[q] : 0.0;
    }
    const bool rowJ = I0 == p0, colJ = K0 == p0;
    if (rowJ && colJ && tid == 0 && drop) atomicAdd(dropped, __popc(drop));
    // T = A_JK (K other than J), X = A_IJ (I other than J)
#pragma unroll
    for (int q = 0; q < 4; q++) {
        T[i][j0 + q] = colJ ? (i == j0 + q ? 1.0 : 0.0) : at(p0, K0, i, j0 + q);
        X[i][j0 + q] = rowJ ? 0.0 : at(I0, p0, i, j0 + q);
    }
    __syncthreads();
    double t[4] = {0.0, 0.0, 0.0, 0.0};  // B A_JK (B itself in column J)
    if (colJ) {
#pragma unroll
        for (int q = 0; q < 4; q++) t[q] = Bs[i][j0 + q];
    } else {
#pragma unroll 8
        for (int s = 0; s < W; s++) {
            const double b = Bs[i][s];
#pragma unroll
            for (int q = 0; q < 4; q++) t[q] = fma(b, T[s][j0 + q], t[q]);
        }
    }
    if (!rowJ) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) T[i][j0 + q] = t[q];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) t[q] = colJ ? 0.0 : at(I0, K0, i, j0 + q);
#pragma unroll 8
        for (int s = 0; s < W; s++) {
            const double x = -X[i][s];
#pragma unroll
            for (int q = 0; q < 4; q++) t[q] = fma(x, T[s][j0 + q], t[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (I0 + i < C && K0 + j0 + q < C) out[(size_t)(I0 + i) * C + K0 + j0 + q] = t[q];
}

// Part rows of A_c^-1: out64/out32[r][k] = Ainv[src[r]][k].
__global__ void coarse_rows_kernel(int rows, int C, const int* __restrict__ src, const double* __restrict__ Ainv,
                                   double* __restrict__ out64, float* __restrict__ out32) {
    const long total = (long)rows * C;
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < total; q += (long)gridDim.x * blockDim.x) {
        const int r = (int)(q / C), k = (int)(q - (long)r * C);
        const double v = Ainv[(size_t)src[r] * C + k];
        out64[q] = v;
        out32[q] = (float)v;
    }
}

}  // namespace pg
