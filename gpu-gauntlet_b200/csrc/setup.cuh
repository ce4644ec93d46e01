// Device kernels of a plan's set-up and of the small steps around a solve.
//
//   ke_kernel          element stiffness, FP64 (and an FP32 copy), per element
//   binv_kernel        3x3 block diagonal, constrained rule, FP64 inversion
//   row_fill_kernel    the assembled row blocks the PCG kernels read (rows.cuh)
//   applyk_color_kernel, bc_copy_kernel
//                      y = K x colour by colour (test hook, reference layout;
//                      also the FP64 K x of the correction steps)
//   power_start_kernel, power_step_kernel, two_norms_kernel
//                      lambda_max(D^-1 K) power steps for the Chebyshev smoother
//   residual_*_kernel, add_kernel
//                      FP64 correction after a stagnated mixed solve
//   elem_moments_kernel, node_moments_kernel
//                      nodal bending moments
#pragma once

#include <cstdint>

#include "element.cuh"
#include "rows.cuh"

namespace pg {

template <int NPE>
__global__ void ke_kernel(int Ne, const float* __restrict__ nodes,
                          const uint32_t* __restrict__ elements, double E, double nu, double t,
                          const float* __restrict__ elem_t, double* __restrict__ ke64,
                          float* __restrict__ ke32) {
    constexpr int KK = 9 * NPE * NPE;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= Ne) return;
    double c[2 * NPE];
#pragma unroll
    for (int k = 0; k < NPE; k++) {
        const uint32_t n = elements[(size_t)e * NPE + k];
        c[2 * k] = nodes[2 * n];
        c[2 * k + 1] = nodes[2 * n + 1];
    }
    const double te = elem_t ? (double)elem_t[e] : t;
    double Ke[KK];
    if constexpr (NPE == 4)
        q4_ke(c, E, nu, te, Ke);
    else
        dkt_ke(c, E, nu, te, Ke);
    for (int i = 0; i < KK; i++) {
        ke64[(size_t)e * KK + i] = Ke[i];
        if (ke32) ke32[(size_t)e * KK + i] = (float)Ke[i];
    }
}

// computeBlockDiagonal + invertBlockDiagonal (solver.ts:188-304), per node.
__global__ void binv_kernel(int Nn, int npe, const int* __restrict__ inc_ptr,
                            const int* __restrict__ inc_idx, const double* __restrict__ ke64,
                            const uint8_t* __restrict__ cons, double* __restrict__ binv64,
                            float* __restrict__ binv32) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Nn) return;
    const int nd = 3 * npe, kk = nd * nd;
    double b[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int q = inc_ptr[n]; q < inc_ptr[n + 1]; q++) {
        const int e = inc_idx[q] >> 2, k = inc_idx[q] & 3;
        const double* K = ke64 + (size_t)e * kk;
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) b[r * 3 + c] += K[(3 * k + r) * nd + 3 * k + c];
    }
    const bool wc = cons[3 * n], xc = cons[3 * n + 1], yc = cons[3 * n + 2];
    double o[9];
    bool ident = wc && xc && yc;
    if (!ident) {
        if (wc) { b[0] = 1; b[1] = 0; b[2] = 0; b[3] = 0; b[6] = 0; }
        if (xc) { b[4] = 1; b[1] = 0; b[7] = 0; b[3] = 0; b[5] = 0; }
        if (yc) { b[8] = 1; b[2] = 0; b[5] = 0; b[6] = 0; b[7] = 0; }
        const double a00 = b[0], a01 = b[1], a02 = b[2], a10 = b[3], a11 = b[4], a12 = b[5];
        const double a20 = b[6], a21 = b[7], a22 = b[8];
        const double det = a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) +
                           a02 * (a10 * a21 - a11 * a20);
        if (fabs(det) < 1e-30) {
            ident = true;
        } else {
            const double id = 1.0 / det;
            o[0] = id * (a11 * a22 - a12 * a21);
            o[1] = id * (a02 * a21 - a01 * a22);
            o[2] = id * (a01 * a12 - a02 * a11);
            o[3] = id * (a12 * a20 - a10 * a22);
            o[4] = id * (a00 * a22 - a02 * a20);
            o[5] = id * (a02 * a10 - a00 * a12);
            o[6] = id * (a10 * a21 - a11 * a20);
            o[7] = id * (a01 * a20 - a00 * a21);
            o[8] = id * (a00 * a11 - a01 * a10);
        }
    }
    for (int i = 0; i < 9; i++) {
        const double v = ident ? ((i % 4 == 0) ? 1.0 : 0.0) : o[i];
        binv64[(size_t)n * 9 + i] = v;
        if (binv32) binv32[(size_t)n * 9 + i] = (float)v;
    }
}

// One colour of y += K x (elements of a colour share no node: no atomics).
__global__ void applyk_color_kernel(int cnt, const uint32_t* __restrict__ list, int npe,
                                    const uint32_t* __restrict__ elements,
                                    const double* __restrict__ ke64, const double* __restrict__ x,
                                    double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    const uint32_t e = list[i];
    const int nd = 3 * npe;
    int dof[12];
    double xl[12];
    for (int k = 0; k < npe; k++)
        for (int d = 0; d < 3; d++) {
            dof[3 * k + d] = (int)elements[(size_t)e * npe + k] * 3 + d;
            xl[3 * k + d] = x[dof[3 * k + d]];
        }
    const double* K = ke64 + (size_t)e * nd * nd;
    for (int r = 0; r < nd; r++) {
        double s = 0;
        for (int c = 0; c < nd; c++) s += K[r * nd + c] * xl[c];
        y[dof[r]] += s;
    }
}

__global__ void bc_copy_kernel(int n, const uint8_t* __restrict__ cons,
                               const double* __restrict__ x, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && cons[i]) y[i] = x[i];
}

// Start vector of the lambda_max(D^-1 K) power iteration: 1 + 0.5 sin(0.7 i),
// 0 on constrained DOFs.
__global__ void power_start_kernel(int n, const uint8_t* __restrict__ cons, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = cons[i] ? 0.0 : 1.0 + 0.5 * sin(0.7 * (double)i);
}

// One power step z = D^-1 K x on the owned rows of part blockIdx.x (row blocks
// from memory, one warp a group of 10 rows; constrained rows the identity).
// Bound by reading the row blocks from L2 (13 MB on the 60k-DOF plate, 27 us a
// step when it gathered from the 23 MB of element matrices node by node).
__global__ void power_step_kernel(const int* __restrict__ node_off, const int* __restrict__ nown,
                                  const int* __restrict__ nodes, const int* __restrict__ grp_off,
                                  const int* __restrict__ grp_q, const uint16_t* __restrict__ rcol,
                                  const double* __restrict__ rk64, const uint8_t* __restrict__ cons,
                                  const double* __restrict__ binv, const double* __restrict__ x,
                                  double* __restrict__ z) {
    const int g = blockIdx.x, n0 = node_off[g], no = nown[g], gb = grp_off[g];
    const int lane = threadIdx.x & 31, d = lane % 3, nw = (int)(blockDim.x >> 5);
    for (int grp = blockIdx.y * nw + (int)(threadIdx.x >> 5); grp * kRowGroup < no; grp += gridDim.y * nw) {
        const int i = grp * kRowGroup + lane / 3;
        const bool live = lane < kRowLanes && i < no;
        double s[3] = {0.0, 0.0, 0.0};
        if (lane < kRowLanes) {
            const int q1 = grp_q[gb + grp + 1];
#pragma unroll 3
            for (int q = grp_q[gb + grp]; q < q1; q++) {
                const double* v = x + 3 * (size_t)nodes[n0 + rcol[(size_t)q * kRowLanes + lane]];
                const double* b = rk64 + (size_t)q * 9 * kRowLanes + lane;
#pragma unroll
                for (int r = 0; r < 3; r++)
                    s[r] = fma(b[(3 * r + 2) * kRowLanes], v[2],
                               fma(b[(3 * r + 1) * kRowLanes], v[1], fma(b[3 * r * kRowLanes], v[0], s[r])));
            }
        }
        double y = row_join(s);
        double b[3] = {0.0, 0.0, 0.0};
        const int k = live ? 3 * nodes[n0 + i] + d : 0;
        if (live) {
            if (cons[k]) y = x[k];
#pragma unroll
            for (int q = 0; q < 3; q++) b[q] = binv[3 * (size_t)k + (d + q) % 3];
        }
        y = jacobi_lane(b, y);
        if (live) z[k] = y;
    }
}

// out[0] = |a|^2, out[1] = |b|^2.  One block of 1024 threads (a fixed order of
// additions).
__global__ void two_norms_kernel(int n, const double* __restrict__ a, const double* __restrict__ b, double* out) {
    __shared__ double red[2][32];
    double s = 0.0, t = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += 1024) {
        s = fma(a[i], a[i], s);
        t = fma(b[i], b[i], t);
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = s;
        red[1][threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double v = 0.0;
        for (int w = 0; w < 32; w++) v += red[threadIdx.x][w];
        out[threadIdx.x] = v;
    }
}

// r = F - y narrowed to FP32, 0 on constrained rows (y = K x): the load of
// an FP64 correction solve K d = F - K x.  r may be F itself.
__global__ void residual_f32_kernel(int n, const uint8_t* cons, const float* F, const double* y, float* r) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = cons[i] ? 0.0f : (float)((double)F[i] - y[i]);
}

// x += a
__global__ void add_kernel(int n, const double* __restrict__ a, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += a[i];
}

// out[0] += sum (F - y)^2, out[1] += sum F^2 over the unconstrained rows
// (y = K x): the true residual of x.  out must start at zero.
__global__ void residual_norms_kernel(int n, const uint8_t* __restrict__ cons, const float* __restrict__ F,
                                      const double* __restrict__ y, double* out) {
    double a = 0.0, b = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (!cons[i]) {
            const double f = (double)F[i], r = f - y[i];
            a += r * r;
            b += f * f;
        }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, a);
        atomicAdd(out + 1, b);
    }
}

// Local index of global node m in a part: three runs of ascending node ids,
// the owned nodes [0, no), ring 1 [no, n1) and the rest [n1, nloc) (one halo
// ring: n1 = no).
__device__ __forceinline__ int local_index(const int* __restrict__ nodes, int no, int n1, int nloc, int m) {
    const int seg[4] = {0, no, n1, nloc};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        int lo = seg[k], hi = seg[k + 1];
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (nodes[mid] < m) lo = mid + 1;
            else hi = mid;
        }
        if (lo < seg[k + 1] && nodes[lo] == m) return lo;
    }
    return 0;
}

// Columns and blocks of every part's rows from the element matrices: one
// thread per (row, slot residue), blockIdx.x the part, blockIdx.y a share of
// its groups.
template <int NPE>
__global__ void row_fill_kernel(const int* __restrict__ node_off, const int* __restrict__ nown,
                                const int* __restrict__ n1, const int* __restrict__ nodes,
                                const int* __restrict__ grp_off, const int* __restrict__ grp_q,
                                const int* __restrict__ inc_ptr, const int* __restrict__ inc_idx,
                                const uint32_t* __restrict__ elements, const double* __restrict__ ke64,
                                uint16_t* __restrict__ rcol, double* __restrict__ rk64,
                                float* __restrict__ rk32) {
    constexpr int ND = 3 * NPE;
    const int g = blockIdx.x, n0 = node_off[g], nloc = node_off[g + 1] - n0, no = nown[g], nn1 = n1[g];
    const int gb = grp_off[g], ng = grp_off[g + 1] - gb;
    const int* pn = nodes + n0;
    for (int t = blockIdx.y * blockDim.x + threadIdx.x; t < ng * kRowLanes; t += gridDim.y * blockDim.x) {
        const int grp = t / kRowLanes, lane = t - grp * kRowLanes, i = grp * kRowGroup + lane / 3, d = lane % 3;
        const int q0 = grp_q[gb + grp], q1 = grp_q[gb + grp + 1];
        int q = q0;
        if (i < nn1) {
            const int n = pn[i], a = inc_ptr[n], b = inc_ptr[n + 1];
            int prev = -1;
            for (int j = 0;; j++) {
                // the next node id of the row: the smallest above the last
                int m = 0x7fffffff;
                for (int k = a; k < b; k++) {
                    const uint32_t* en = elements + (size_t)(inc_idx[k] >> 2) * NPE;
#pragma unroll
                    for (int p = 0; p < NPE; p++) {
                        const int v = (int)en[p];
                        if (v > prev && v < m) m = v;
                    }
                }
                if (m == 0x7fffffff) break;
                prev = m;
                if (j % 3 != d) continue;
                double blk[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
                for (int k = a; k < b; k++) {
                    const int e = inc_idx[k] >> 2;
                    const double* K = ke64 + (size_t)e * ND * ND + 3 * (inc_idx[k] & 3) * ND;
#pragma unroll
                    for (int p = 0; p < NPE; p++)
                        if ((int)elements[(size_t)e * NPE + p] == m)
#pragma unroll
                            for (int r = 0; r < 9; r++) blk[r] += K[(r / 3) * ND + 3 * p + r % 3];
                }
                rcol[(size_t)q * kRowLanes + lane] = (uint16_t)local_index(pn, no, nn1, nloc, m);
#pragma unroll
                for (int r = 0; r < 9; r++) {
                    const size_t o = ((size_t)q * 9 + r) * kRowLanes + lane;
                    rk64[o] = blk[r];
                    rk32[o] = (float)blk[r];
                }
                q++;
            }
        }
        for (; q < q1; q++) {  // padding: a zero block on the row itself
            rcol[(size_t)q * kRowLanes + lane] = (uint16_t)(i < nn1 ? i : 0);
            for (int r = 0; r < 9; r++) {
                const size_t o = ((size_t)q * 9 + r) * kRowLanes + lane;
                rk64[o] = 0.0;
                rk32[o] = 0.0f;
            }
        }
    }
}

// shared[n] = 1 for every node that is a ghost of some part.
__global__ void mark_ghosts_kernel(const int* __restrict__ node_off, const int* __restrict__ nown,
                                   const int* __restrict__ nodes, uint8_t* __restrict__ shared) {
    const int g = blockIdx.x;
    for (int i = node_off[g] + nown[g] + threadIdx.x; i < node_off[g + 1]; i += blockDim.x) shared[nodes[i]] = 1;
}

// Bending moments at each element's centroid (postprocess.ts:59-264):
// curvatures from the rotations (Q4: shape derivatives at xi = eta = 0
// through the Jacobian; DKT: linear-triangle derivatives), M = D (k_x +
// nu k_y, k_y + nu k_x, (1 - nu) k_xy / 2) with the plate's uniform D.
// em[e] = {Mx, My, Mxy, weight}; weight 0 marks a degenerate triangle
// (|2A| < 1e-15), which the reference leaves out of the nodal averages.
template <int NPE>
__global__ void elem_moments_kernel(int Ne, const float* __restrict__ nodes,
                                    const uint32_t* __restrict__ el, double D, double nu,
                                    const double* __restrict__ x, double4* __restrict__ em) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= Ne) return;
    const uint32_t* en = el + (size_t)e * NPE;
    double dNdx[NPE], dNdy[NPE];
    if constexpr (NPE == 4) {
        const double dXi[4] = {-0.25, 0.25, 0.25, -0.25}, dEta[4] = {-0.25, -0.25, 0.25, 0.25};
        double J11 = 0, J12 = 0, J21 = 0, J22 = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double xi = nodes[2 * en[i]], yi = nodes[2 * en[i] + 1];
            J11 += dXi[i] * xi;
            J12 += dXi[i] * yi;
            J21 += dEta[i] * xi;
            J22 += dEta[i] * yi;
        }
        const double inv = 1.0 / (J11 * J22 - J12 * J21);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            dNdx[i] = inv * (J22 * dXi[i] - J12 * dEta[i]);
            dNdy[i] = inv * (-J21 * dXi[i] + J11 * dEta[i]);
        }
    } else {
        const double x1 = nodes[2 * en[0]], y1 = nodes[2 * en[0] + 1];
        const double x2 = nodes[2 * en[1]], y2 = nodes[2 * en[1] + 1];
        const double x3 = nodes[2 * en[2]], y3 = nodes[2 * en[2] + 1];
        const double twoA = (x2 - x1) * (y3 - y1) - (x3 - x1) * (y2 - y1);
        if (fabs(twoA) < 1e-15) {
            em[e] = make_double4(0.0, 0.0, 0.0, 0.0);
            return;
        }
        const double inv = 1.0 / twoA;
        dNdx[0] = (y2 - y3) * inv; dNdy[0] = (x3 - x2) * inv;
        dNdx[1] = (y3 - y1) * inv; dNdy[1] = (x1 - x3) * inv;
        dNdx[2] = (y1 - y2) * inv; dNdy[2] = (x2 - x1) * inv;
    }
    double kx = 0, ky = 0, kxy = 0;
#pragma unroll
    for (int i = 0; i < NPE; i++) {
        const double tx = x[3 * (size_t)en[i] + 1], ty = x[3 * (size_t)en[i] + 2];
        kx += dNdx[i] * ty;
        ky += -dNdy[i] * tx;
        kxy += dNdy[i] * ty - dNdx[i] * tx;
    }
    em[e] = make_double4(D * (kx + nu * ky), D * (ky + nu * kx), D * (1 - nu) * kxy / 2, 1.0);
}

// Nodal averages of the element moments, summed in element order over each
// node's incidence list (postprocess.ts:132-155).  M: [3][Nn] Mx, My, Mxy.
__global__ void node_moments_kernel(int Nn, const int* __restrict__ inc_ptr,
                                    const int* __restrict__ inc_idx, const double4* __restrict__ em,
                                    double* __restrict__ M) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Nn) return;
    double sx = 0, sy = 0, sxy = 0, c = 0;
    for (int q = inc_ptr[n]; q < inc_ptr[n + 1]; q++) {
        const double4 m = em[inc_idx[q] / 4];
        if (m.w == 0.0) continue;
        sx += m.x;
        sy += m.y;
        sxy += m.z;
        c += 1.0;
    }
    M[n] = c > 0 ? sx / c : 0.0;
    M[Nn + n] = c > 0 ? sy / c : 0.0;
    M[2 * (size_t)Nn + n] = c > 0 ? sxy / c : 0.0;
}

}  // namespace pg
