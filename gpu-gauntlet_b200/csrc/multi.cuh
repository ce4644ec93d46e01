// Load cases of one plate solved together: NR right-hand sides of the same
// operator advance in lockstep through one persistent launch.
//
// Every per-DOF vector of the single solve (r, u, p, s, w, x and the row
// products) holds NR values per DOF, case-interleaved ([dof][case]), so the
// product reads each row block once for NR vectors (rows.cuh; a warp's first
// group of rows from registers) and the
// coarse correction applies each A_c^-1 row to NR restrictions.  One
// exchange round per iteration carries every case's partial sums and ghost
// values, so the grid-wide wait -- the dominant cost of a single 60k-DOF
// solve -- is paid once for NR cases.
//
// Each case keeps its own PCG scalars (alpha, beta, stop state, residual
// reference), decided by lane `case` of warp 0.  A case that has stopped
// continues with alpha = beta = 0, which leaves its x, r and coarse state
// unchanged.  In mixed precision a residual replacement runs when any case
// asks for one: the round computes every case's FP64 residual, but only the
// cases that asked replace r and their coarse state (the others keep their
// recurrences untouched and only use the true residual for an early
// convergence test).
//
// The 3 NR dot products are polled and summed by warps of their own while the
// others take the ghosts and the coarse restrictions, with the addresses'
// divisions by constants: four cases of the 60k-DOF plate (mixed two-level
// Chebyshev) went from 26.1 to 15.8 us per iteration, two from 11.4 to 10.8.
//
// Threads of the case-interleaved loops handle item q = (dof or node) * NR +
// case with a block size that is a multiple of NR, so each thread works on
// one case (threadIdx.x % NR) throughout.
#pragma once

#include "kernels.cuh"

namespace pg {

// Words of one block's partial-sum slot: up to 6 sums per case, 2 tagged
// words per FP64 sum, in 128-byte lines of its own (see kRep).
template <int NR>
constexpr int multi_slot_words() { return (2 * 6 * NR + 15) / 16 * 16; }

// NR consecutive values (one per case) as one aligned access.
template <typename T, int NR>
struct alignas(sizeof(T) * NR <= 16 ? sizeof(T) * NR : 16) CaseVec {
    T v[NR];
};

// v -= o, case by case
template <typename T, int NR>
__device__ __forceinline__ void case_sub(CaseVec<T, NR>& v, const CaseVec<T, NR>& o) {
#pragma unroll
    for (int i = 0; i < NR; i++) v.v[i] -= o.v[i];
}

// s[r][k] += the blocks of q-steps [0, steps) at b (lane offset included) times
// case k of u at the columns c, its w less w0 (0, or the row's own w; FP32
// only).
template <typename T, int NR>
__device__ __forceinline__ void row_steps_multi(const T* __restrict__ u, const uint16_t* __restrict__ c,
                                                const T* __restrict__ k, int steps, const CaseVec<T, NR>& w0,
                                                T (&s)[3][NR]) {
    using V = CaseVec<T, NR>;
#pragma unroll 1
    for (int q = 0; q < steps; q++) {
        const V* v = reinterpret_cast<const V*>(u) + 3 * (int)c[q * kRowLanes];
        V v0 = v[0];
        const V v1 = v[1], v2 = v[2];
        if constexpr (sizeof(T) == 4) case_sub(v0, w0);
        const T* b = k + q * 9 * kRowLanes;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const T k0 = b[3 * r * kRowLanes], k1 = b[(3 * r + 1) * kRowLanes], k2 = b[(3 * r + 2) * kRowLanes];
#pragma unroll
            for (int i = 0; i < NR; i++) s[r][i] = fma(k2, v2.v[i], fma(k1, v1.v[i], fma(k0, v0.v[i], s[r][i])));
        }
    }
}

// Writes the rows' products of one group to y ([3 rows][case]): lane 3 i + d
// gets component d of row i of every case (rows.cuh).
template <typename T, int NR>
__device__ __forceinline__ void join_store(const T (&s)[3][NR], T* __restrict__ y, int grp, int nrows) {
    const int lane = threadIdx.x & 31, n = grp * kRowGroup + lane / 3;
    CaseVec<T, NR> o;
#pragma unroll
    for (int i = 0; i < NR; i++) {
        const T si[3] = {s[0][i], s[1][i], s[2][i]};
        o.v[i] = row_join(si);
    }
    if (lane < kRowLanes && n < nrows) reinterpret_cast<CaseVec<T, NR>*>(y)[3 * n + lane % 3] = o;
}

// y = K u on the part's first nrows rows for NR case-interleaved vectors, one
// warp a group of rows; each block entry is read once for all cases, a warp's
// first group from registers.
template <typename T, int NR>
__device__ __forceinline__ void rows_multi(const RegRows<T>& R, const RowMem<T>& A, const T* __restrict__ u,
                                           T* __restrict__ y, int nrows, int w_rigid) {
    using V = CaseVec<T, NR>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int grp = warp; grp * kRowGroup < nrows; grp += nw) {
        T s[3][NR];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int i = 0; i < NR; i++) s[r][i] = T(0);
        V w0{};
        const int own = grp * kRowGroup + lane / 3;
        if (sizeof(T) == 4 && w_rigid && lane < kRowLanes && own < nrows) w0 = reinterpret_cast<const V*>(u)[3 * own];
        const int q0 = A.gq[grp], w = A.gq[grp + 1] - q0;
        int done = 0;
        if (grp == warp) {
            done = kRegSteps;
#pragma unroll
            for (int q = 0; q < kRegSteps; q++) {
                const V* v = reinterpret_cast<const V*>(u) + R.c[q];
                V v0 = v[0];
                const V v1 = v[1], v2 = v[2];
                if constexpr (sizeof(T) == 4) case_sub(v0, w0);
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int i = 0; i < NR; i++)
                        s[r][i] = fma(R.k[9 * q + 3 * r + 2], v2.v[i],
                                      fma(R.k[9 * q + 3 * r + 1], v1.v[i], fma(R.k[9 * q + 3 * r], v0.v[i], s[r][i])));
            }
        }
        if (done < w && lane < kRowLanes) {
            const int g0 = A.go[grp];
            const uint16_t* cq = A.col + (q0 + done) * kRowLanes + lane;
            if (g0 >= 0)
                row_steps_multi<T, NR>(u, cq, A.ks + g0 * 9 * kRowLanes + lane, w - done, w0, s);
            else
                row_steps_multi<T, NR>(u, cq, A.kg + (size_t)(q0 + done) * 9 * kRowLanes + lane, w - done, w0, s);
        }
        join_store<T, NR>(s, y, grp, nrows);
    }
}

// The same in FP64 from global memory (the true residuals of mixed solves).
template <int NR>
__device__ __forceinline__ void rows_multi64(const int* __restrict__ gq, const uint16_t* __restrict__ col,
                                             const double* __restrict__ kg, const double* __restrict__ u,
                                             double* __restrict__ y, int nrows) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int grp = warp; grp * kRowGroup < nrows; grp += nw) {
        double s[3][NR];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int i = 0; i < NR; i++) s[r][i] = 0.0;
        const int q0 = gq[grp];
        if (lane < kRowLanes)
            row_steps_multi<double, NR>(u, col + q0 * kRowLanes + lane, kg + (size_t)q0 * 9 * kRowLanes + lane,
                                        gq[grp + 1] - q0, CaseVec<double, NR>{}, s);
        join_store<double, NR>(s, y, grp, nrows);
    }
}

// Block totals of KP sums per case (each thread holds the KP sums of its
// case threadIdx.x % NR), published as this block's partial sums: value
// m * NR + k of block g goes to every replica r < kRep at words
// pb[(r * G + g) * SW + 2 (m * NR + k)].  All threads call it; one barrier,
// then warp 0 alone works, so `red` must not be written again before a
// later barrier.
template <int NR, int KP>
__device__ void block_publish_multi(double (&v)[KP], double* red, unsigned long long* pb, int G, int g,
                                    unsigned f) {
    constexpr int SW = multi_slot_words<NR>(), K = KP * NR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int m = 0; m < KP; m++)
#pragma unroll
        for (int o = 16; o >= NR; o >>= 1) v[m] += __shfl_xor_sync(0xffffffffu, v[m], o);
    if (lane < NR)
#pragma unroll
        for (int m = 0; m < KP; m++) red[warp * K + m * NR + lane] = v[m];
    __syncthreads();
    if (warp != 0 || lane >= K) return;
    double t = 0.0;
    for (int w = 0; w < nw; w++) t += red[w * K + lane];
#pragma unroll
    for (int r = 0; r < kRep; r++) Tag<double>::put(pb + ((size_t)r * G + g) * SW + 2 * lane, t, f);
}

// This thread's items t, t + stride, ... of an exchange round for NR cases: case k
// of each ghost DOF of vector buffer vb (words ((dof * NR + k) * TW)), to
// dst[dof_local * NR + k] for local DOFs [3 no, 3 nloc), then values K0 .. K0 +
// K - 1 of every block's partial sums, to put(b * K + i, value).  The ghosts
// come first (their owners publish them before their partial sums); S items in
// flight, a slot takes its next item as soon as its item has arrived.  False
// if a wait gave up.
template <typename T, int NR, int K0, int K, int S, typename Put>
__device__ __forceinline__ bool poll_multi(const unsigned long long* __restrict__ pb, int G,
                                           const unsigned long long* __restrict__ vb, T* dst, int no, int nloc,
                                           const int* __restrict__ gid, int g, unsigned f, int t, int stride,
                                           Waiter& wt, Put put) {
    constexpr int TW = Tag<T>::W, SW = multi_slot_words<NR>();
    const int ng = 3 * (nloc - no) * NR, n = ng + G * K;
    pb += (size_t)(g % kRep) * G * SW + 2 * K0;
    auto addr = [&](int i) -> const unsigned long long* {
        if (i < ng) {
            const int k3 = 3 * no + i / NR;
            return vb + ((size_t)(3 * gid[k3 / 3] + k3 % 3) * NR + i % NR) * TW;
        }
        const int q = i - ng;
        return pb + (size_t)(q / (K > 0 ? K : 1)) * SW + 2 * (q % (K > 0 ? K : 1));
    };
    int it[S];
    const unsigned long long* pp[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
        it[s] = t + s * stride;
        pp[s] = it[s] < n ? addr(it[s]) : nullptr;
    }
    int next = t + S * stride;
    wt.spins = 0;
    for (;;) {
        unsigned long long lo[S], hi[S];
        bool any = false;
#pragma unroll
        for (int s = 0; s < S; s++) {
            lo[s] = hi[s] = 0;
            if (it[s] >= n) continue;
            any = true;
            if (it[s] >= ng || TW == 2) {
                ld_relaxed2(pp[s], lo[s], hi[s]);
            } else {
                lo[s] = ld_relaxed(pp[s]);
                hi[s] = lo[s];
            }
        }
        if (!any) return true;
        bool moved = false;
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (it[s] >= n) continue;
            if ((unsigned)(lo[s] >> 32) != f || (unsigned)(hi[s] >> 32) != f) continue;
            const int i = it[s];
            const double v = __longlong_as_double((long long)((hi[s] << 32) | (lo[s] & 0xffffffffull)));
            if (i >= ng) {
                put(i - ng, v);
            } else if constexpr (TW == 2) {
                dst[3 * no * NR + i] = (T)v;
            } else {
                dst[3 * no * NR + i] = (T)__uint_as_float((unsigned)lo[s]);
            }
            it[s] = next;
            next += stride;
            pp[s] = it[s] < n ? addr(it[s]) : nullptr;
            moved = true;
        }
        if (!moved && !wt.keep_going()) return false;
    }
}

// One exchange round by all threads: the first K partial sums of every block
// (staged to sp[G][K]) and the ghost values.
template <typename T, int NR, int K>
__device__ bool exchange_round_multi(const unsigned long long* __restrict__ pb, int G,
                                     const unsigned long long* __restrict__ vb, T* dst, int no, int nloc,
                                     const int* __restrict__ gid, int g, unsigned f, double* sp, Waiter& wt) {
    return poll_multi<T, NR, 0, K, 4>(pb, G, vb, dst, no, nloc, gid, g, f, threadIdx.x, blockDim.x, wt,
                                      [&](int i, double v) { sp[i] = v; });
}

// out[q * NR + k] = sum_j Ai[q][j] y_j^(k) for the part's coarse rows; y [C][NR]
// in the rows' type.  Warps w0.. take two rows each, 16 lanes a row, fixed
// order.  Only the cases in `mask` are written.
template <typename T, int NR>
__device__ __forceinline__ void coarse_apply_multi(const T* __restrict__ Ai, int C, int rows, const T* __restrict__ y,
                                                   double* __restrict__ out, int w0, unsigned mask = 0xffffffffu) {
    using V = CaseVec<T, NR>;
    const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5) - w0;
    const int nw = (int)(blockDim.x >> 5) - w0;
    if (warp < 0) return;
    const int half = lane >> 4, hl = lane & 15;
    for (int q0 = 2 * warp; q0 < rows; q0 += 2 * nw) {
        const int q = q0 + half;
        T acc[2][NR];
#pragma unroll
        for (int k = 0; k < NR; k++) acc[0][k] = acc[1][k] = T(0);
        if (q < rows) {
            const T* row = Ai + (size_t)q * C;
            const V* yv = reinterpret_cast<const V*>(y);
            int j = hl;
#pragma unroll 4
            for (; j + 16 < C; j += 32) {
                const V y0 = yv[j], y1 = yv[j + 16];
                const T m0 = row[j], m1 = row[j + 16];
#pragma unroll
                for (int k = 0; k < NR; k++) {
                    acc[0][k] = fma(m0, y0.v[k], acc[0][k]);
                    acc[1][k] = fma(m1, y1.v[k], acc[1][k]);
                }
            }
            if (j < C) {
                const V y0 = yv[j];
#pragma unroll
                for (int k = 0; k < NR; k++) acc[0][k] = fma(row[j], y0.v[k], acc[0][k]);
            }
        }
#pragma unroll
        for (int k = 0; k < NR; k++) {
            double s = (double)acc[0][k] + (double)acc[1][k];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (hl == 0 && q < rows && ((mask >> k) & 1u)) out[q * NR + k] = s;
        }
    }
}

// ct[(3 b + m) NR + k] = (T) sp[b stride + off + m NR + k]: a round's
// restrictions in the type of the A_c^-1 rows (all threads; a barrier before
// and after is the caller's).
template <typename T, int NR>
__device__ __forceinline__ void stage_coarse(const double* __restrict__ sp, int G, int stride, int off, T* __restrict__ ct) {
    for (int i = threadIdx.x; i < 3 * NR * G; i += blockDim.x) {
        const int b = i / (3 * NR);
        ct[i] = (T)sp[b * stride + off + i - b * 3 * NR];
    }
}

// Per-case decision state (lane k of warp 0 holds case k's).
struct CaseState {
    double inv_gamma, inv_alpha, bnorm, rn_ref, thr_rel, thr_ru, best_trn, final_res, true_rel;
    int xupd, xupd_ref, nru, stall, stop, status;
    bool first, done, asked;
};

template <typename T, bool MIXED, int NR>
__device__ __forceinline__ void pcg_multi_body(const PcgArgs& a, const int g, unsigned char* sm) {
    constexpr int TW = Tag<T>::W, SW = multi_slot_words<NR>();
    const SmemLayout& L = a.L;
    const int tid = threadIdx.x, nt = blockDim.x, kc = tid % NR;
    const int lane = tid & 31;
    const int n0 = a.node_off[g], nloc = a.node_off[g + 1] - n0, no = a.nown[g];
    const int nn1 = a.n1[g];
    const int gb = a.grp_off[g], ng1 = a.grp_off[g + 1] - gb, qb = a.grp_q[gb];
    const int warp = tid >> 5, nw = nt >> 5;
    const bool cheb = a.smoother == 1;
    const T ca = (T)a.cheb_a, cbc = (T)a.cheb_b;
    const size_t N3 = 3 * (size_t)a.Nn;

    T* r = (T*)(sm + L.r);
    T* u = (T*)(sm + L.u);
    T* p = (T*)(sm + L.p);
    T* s = (T*)(sm + L.s);
    T* w = (T*)(sm + L.w);
    T* B = (T*)(sm + L.B);
    T* yt = (T*)(sm + L.yt);  // row products, [3 rows][case]
    T* kts = (T*)(sm + L.kt);
    double* x = (double*)(sm + L.x);
    double* red = (double*)(sm + L.red);
    double* scal = (double*)(sm + L.scal);  // [0, 3NR) dots, [3NR, 4NR) alpha, [4NR, 5NR) beta
    double* sp = (double*)(sm + L.sp);
    int* gid = (int*)(sm + L.gid);
    int* gq = (int*)(sm + L.gq);
    int* go = (int*)(sm + L.go);
    uint16_t* rcol = (uint16_t*)(sm + L.rcol);
    unsigned char* cm = (unsigned char*)(sm + L.cm);
    double* qw = (double*)(sm + L.qw);
    double* csb = (double*)(sm + L.cs);
    double* cvb = (double*)(sm + L.cv);
    int* ctl = (int*)(sm + L.ctl);  // [0] action, [1] final residuals needed, [2] cases replacing r, [3] a wait gave up
    T* nb = (T*)(sm + L.nb);
    int* nslot = (int*)(sm + L.nslot);
    const int rows = a.coarse ? 3 * (a.cagg_off[g + 1] - a.cagg_off[g]) : 0;
    const int RN = rows * NR;
    const T* aig = a.coarse ? (MIXED ? (const T*)a.ainv32 : (const T*)a.ainv64) + (size_t)a.ainv_off[g] * a.C
                            : nullptr;
    T* ais = (T*)(sm + L.ainv);
    T* ct = (T*)(sm + L.ct);  // a round's restrictions [C][NR]
    const T* Ai = a.ainv_smem ? (const T*)ais : aig;
    // FP64 views for the true residual: own arrays in MIXED mode (ytd may
    // share the yt / w / u space), the (then dead) p / yt arrays in FP64
    double* xl = MIXED ? (double*)(sm + L.xl) : (double*)p;
    double* ytd = MIXED ? (double*)(sm + L.ytd) : (double*)yt;
    const T* kg = (MIXED ? (const T*)a.rk32 : (const T*)a.rk64) + (size_t)qb * 9 * kRowLanes;
    const double* kg64 = a.rk64 + (size_t)qb * 9 * kRowLanes;
    const T* Bg = MIXED ? (const T*)a.binv32 : (const T*)a.binv64;

    // ---- load the part ----
    for (int i = tid; i < nloc; i += nt) gid[i] = a.nodes[n0 + i];
    for (int i = tid; i <= ng1; i += nt) gq[i] = a.grp_q[gb + i] - qb;
    __syncthreads();
    if (tid == 0) {
        ctl[3] = 0;
        // the q-steps not in registers go to shared memory while they fit
        int used = 0;
        for (int k = 0; k < ng1; k++) {
            const int need = max(0, gq[k + 1] - gq[k] - (k < nw ? kRegSteps : 0));
            const bool fits = used + need <= L.kq;
            go[k] = fits ? used : -1;
            if (fits) used += need;
        }
    }
    for (int i = tid; i < gq[ng1] * kRowLanes; i += nt) rcol[i] = a.rcol[(size_t)qb * kRowLanes + i];
    if (a.coarse) {
        for (int i = tid; i < nloc; i += nt) {
            nslot[i] = a.node_slot[n0 + i];
#pragma unroll
            for (int q = 0; q < 3; q++) nb[3 * i + q] = (T)a.node_basis[3 * (size_t)(n0 + i) + q];
        }
        for (int j = tid; j < RN; j += nt) csb[j] = 0.0;
        if (a.ainv_smem)
            for (int i = tid; i < rows * a.C; i += nt) ais[i] = aig[i];
    }
    __syncthreads();
    const RowMem<T> A{gq, go, rcol, kts, kg};
    RegRows<T> R;
    {
        const int w0 = warp < ng1 ? gq[warp + 1] - gq[warp] : 0;
#pragma unroll
        for (int q = 0; q < kRegSteps; q++) {
            const bool has = q < w0 && lane < kRowLanes;
            const size_t o = has ? (size_t)(gq[warp] + q) : 0;
            R.c[q] = has ? 3 * (int)rcol[o * kRowLanes + lane] : 0;
#pragma unroll
            for (int k = 0; k < 9; k++) R.k[9 * q + k] = has ? kg[(o * 9 + k) * kRowLanes + lane] : T(0);
        }
    }
    for (int k = warp; k < ng1; k += nw) {
        if (go[k] < 0) continue;
        const int skip = k < nw ? kRegSteps : 0, need = gq[k + 1] - gq[k] - skip;
        const T* src = kg + (size_t)(gq[k] + skip) * 9 * kRowLanes;
        T* dst = kts + go[k] * 9 * kRowLanes;
        for (int i = lane; i < need * 9 * kRowLanes; i += 32) dst[i] = src[i];
    }
    for (int n = tid; n < nloc; n += nt) {
        const int G3 = 3 * gid[n];
#pragma unroll
        for (int d = 0; d < 3; d++) cm[3 * n + d] = a.cons[G3 + d];
#pragma unroll
        for (int q = 0; q < 9; q++) B[9 * n + q] = Bg[(size_t)gid[n] * 9 + q];
    }
    __syncthreads();
    for (int q = tid; q < nloc * NR; q += nt) {
        const int n = q / NR, G3 = 3 * gid[n];
        T rv[3], uv[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const int i = (3 * n + d) * NR + kc;
            rv[d] = cm[3 * n + d] ? T(0) : (T)a.F[kc * N3 + G3 + d];
            r[i] = rv[d];
            p[i] = T(0);
            s[i] = T(0);
            if (n < no) x[i] = 0.0;
        }
        block_jacobi3(B + 9 * n, rv, uv);
#pragma unroll
        for (int d = 0; d < 3; d++) u[(3 * n + d) * NR + kc] = uv[d];
    }
    __syncthreads();

    // u = ca t - cb D^-1 (K t) at node n of case kc (t in u, K t in yt)
    auto smooth = [&](int n) {
        T k3[3], tv[3], v3[3];
#pragma unroll
        for (int d = 0; d < 3; d++) k3[d] = yt[(3 * n + d) * NR + kc];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            tv[d] = u[(3 * n + d) * NR + kc];
            if (cm[3 * n + d]) k3[d] = tv[d];
        }
        block_jacobi3(B + 9 * n, k3, v3);
#pragma unroll
        for (int d = 0; d < 3; d++) u[(3 * n + d) * NR + kc] = ca * tv[d] - cbc * v3[d];
    };
    // u += P c at node n of case kc, c3 = its aggregate's coarse values
    auto prolong = [&](int n, const double* c3) {
        T uv[3];
#pragma unroll
        for (int d = 0; d < 3; d++) uv[d] = u[(3 * n + d) * NR + kc];
        prolong3(c3, cm + 3 * n, nb + 3 * n, uv);
#pragma unroll
        for (int d = 0; d < 3; d++) u[(3 * n + d) * NR + kc] = uv[d];
    };
    if (cheb) {
        rows_multi<T, NR>(R, A, u, yt, nn1, a.w_rigid);
        __syncthreads();
        for (int q = tid; q < nn1 * NR; q += nt) smooth(q / NR);
        __syncthreads();
    }
    PhaseClock clk;
    clk.start(a.timing && g == a.G / 2 && tid == 0, (long long*)(sm + L.clk));
    Waiter wt;
    wt.start(a.timeout_ns, a.abort_flag, &a.res->wait_failures);
    unsigned e = a.tag0 + 1, xe = a.tag0 + 1;
    int status = ST_OK;

    // ---- two-level: u0 += P A_c^-1 P^T r0 for every case ----
    if (a.coarse) {
        double v0[3] = {0.0, 0.0, 0.0};
        for (int q = tid; q < no * NR; q += nt) {
            const int n = q / NR;
            T rv[3];
#pragma unroll
            for (int d = 0; d < 3; d++) rv[d] = r[(3 * n + d) * NR + kc];
            restrict3(rv, cm + 3 * n, nb + 3 * n, v0);
        }
        unsigned long long* pb0 = a.llp + (size_t)(e & 1) * kRep * a.G * SW;
        block_publish_multi<NR, 3>(v0, red, pb0, a.G, g, e);
        const bool ok = exchange_round_multi<T, NR, 3 * NR>(pb0, a.G, nullptr, w, no, no, gid, g, e, sp, wt);
        if (__syncthreads_or(!ok)) {
            status = ST_TIMEOUT;
        } else {
            stage_coarse<T, NR>(sp, a.G, 3 * NR, 0, ct);
            __syncthreads();
            coarse_apply_multi<T, NR>(Ai, a.C, rows, ct, cvb, 0);
            __syncthreads();
            for (int q = tid; q < nloc * NR; q += nt) {
                const int n = q / NR, sl = 3 * nslot[n];
                const double c3[3] = {cvb[sl * NR + kc], cvb[(sl + 1) * NR + kc], cvb[(sl + 2) * NR + kc]};
                prolong(n, c3);
            }
            __syncthreads();
        }
        e++;
    }

    CaseState cs{};
    cs.inv_gamma = 1.0;
    cs.inv_alpha = 1.0;
    cs.best_trn = INFINITY;
    cs.stop = -1;
    cs.true_rel = -1.0;
    cs.first = true;
    const double thr_abs = a.tol * a.tol;
    const unsigned cmask = (1u << NR) - 1u;
    int cb = 0;

    for (int it = 0; status == ST_OK; it++) {
        // ---- w = A u on owned rows, every case ----
        rows_multi<T, NR>(R, A, u, yt, no, a.w_rigid);
        __syncthreads();
        clk.lap(0);
        // ---- BC rows, dot products, publish w ----
        double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        unsigned long long* vb = a.llv + (size_t)(e & 1) * N3 * NR * 2;
        unsigned long long* pb = a.llp + (size_t)(e & 1) * kRep * a.G * SW;
        for (int q = tid; q < 3 * no * NR; q += nt) {
            const int k3 = q / NR, n = k3 / 3, d = k3 - 3 * n;
            T wk = yt[q];
            const bool c = cm[k3] != 0;
            const T uk = u[q], rk = r[q];
            if (c) wk = uk;
            w[q] = wk;
            v[0] += (double)rk * (double)uk;
            v[1] += (double)wk * (double)uk;
            v[2] += (double)rk * (double)rk;
            Tag<T>::put(vb + ((size_t)(3 * gid[n] + d) * NR + kc) * TW, wk, e);
            if (a.coarse && !c) {
                const T* bs = nb + 3 * n;
                const double wd = (double)wk;
                if (d == 0) {
                    v[3] += wd;
                    v[4] += (double)bs[1] * wd;
                    v[5] += (double)bs[0] * wd;
                } else if (d == 1) {
                    v[4] += (double)bs[2] * wd;
                } else {
                    v[5] -= (double)bs[2] * wd;
                }
            }
        }
        clk.lap(1);
        if (a.coarse) {
            block_publish_multi<NR, 6>(v, red, pb, a.G, g, e);
        } else {
            double v3[3] = {v[0], v[1], v[2]};
            block_publish_multi<NR, 3>(v3, red, pb, a.G, g, e);
        }
        clk.lap(2);
        // ---- exchange: warps 0 .. ND - 1 the 3 NR dot products, the others the
        //      ghosts and the coarse restrictions ----
        constexpr int ND = NR == 2 ? 6 : 4;  // NR = 4: three dot products a warp
        if (warp >= ND) {
            const int t = tid - 32 * ND, st = nt - 32 * ND;
            const bool ok = a.coarse
                ? poll_multi<T, NR, 3 * NR, 3 * NR, 4>(pb, a.G, vb, w, no, nloc, gid, g, e, t, st, wt,
                                                       [&](int i, double v) { ct[i] = (T)v; })
                : poll_multi<T, NR, 0, 0, 3>(pb, a.G, vb, w, no, nloc, gid, g, e, t, st, wt, [](int, double) {});
            if (!ok) ctl[3] = 1;
        } else {
            bool ok = true;
            for (int k = warp; k < 3 * NR; k += ND) {
                double d;
                ok = poll_total<SW>(pb, a.G, g, kRep, k, e, d, wt) && ok;
                if (lane == 0) scal[k] = d;
            }
            if (a.test_stall && it == 0 && tid == 0) {
                // the two spare words after the partial-sum buffers: a tag no
                // block writes, so the wait must run out
                double never;
                ok = ok && poll<double>(a.llp + (size_t)2 * kRep * a.G * multi_slot_words<4>(), 0xffffffffu,
                                        never, wt);
            }
            if (!ok) ctl[3] = 1;
            asm volatile("bar.sync 2, %0;" ::"r"(32 * ND) : "memory");
        }
        e++;
        clk.lap(4);
        // ---- decisions: lane k of warp 0 for case k ----
        __syncwarp();
        if (tid < 32) {
            int want = ACT_UPDATE;
            const bool me = lane < NR;
            const double gamma = scal[me ? lane : 0], delta = scal[me ? NR + lane : 0];
            const double rho = scal[me ? 2 * NR + lane : 0];
            if (me && !cs.done) {
                if (!isfinite(gamma) || !isfinite(delta) || !isfinite(rho)) {
                    cs.status = ST_NONFINITE;
                    cs.done = true;
                    cs.stop = STOP_BREAKDOWN;
                    if (g == 0) {
                        a.res[lane].nonfinite_it = it;
                        a.res[lane].nonfinite_vals[0] = gamma;
                        a.res[lane].nonfinite_vals[1] = delta;
                        a.res[lane].nonfinite_vals[2] = rho;
                    }
                } else if (cs.first && rho < 1e-60) {
                    cs.bnorm = sqrt(rho);
                    cs.stop = STOP_ZERO_RHS; cs.final_res = 0.0; cs.true_rel = 0.0; cs.done = true;
                } else {
                    if (cs.first) {
                        cs.bnorm = sqrt(rho);
                        cs.rn_ref = cs.bnorm;
                        cs.thr_rel = a.tol * cs.bnorm * (a.tol * cs.bnorm);
                        cs.thr_ru = a.reliable_delta * cs.rn_ref * (a.reliable_delta * cs.rn_ref);
                    } else {
                        const bool conv = (a.stop_rule == 0 && rho < thr_abs) || rho < cs.thr_rel;
                        if (MIXED && (conv || rho <= cs.thr_ru || cs.xupd - cs.xupd_ref >= a.reliable_interval))
                            want = ACT_RU;
                        else if (!MIXED && conv) {
                            cs.stop = STOP_CONVERGED; cs.final_res = sqrt(rho); cs.done = true;
                        }
                    }
                    if (!cs.done && want == ACT_UPDATE && cs.xupd >= a.maxit) {
                        cs.stop = STOP_MAX_ITER; cs.final_res = sqrt(rho); cs.done = true;
                    }
                }
            }
            const unsigned ru = __ballot_sync(0xffffffffu, me && !cs.done && want == ACT_RU) & cmask;
            const unsigned dn = __ballot_sync(0xffffffffu, me && cs.done) & cmask;
            const int act = ru ? ACT_RU : (dn == cmask ? ACT_STOP : ACT_UPDATE);
            if (me) {
                cs.asked = (ru >> lane) & 1u;
                double alpha = 0.0, beta = 0.0;
                if (act == ACT_UPDATE && !cs.done) {
                    beta = cs.first ? 0.0 : gamma * cs.inv_gamma;
                    const double pap = cs.first ? delta : delta - beta * gamma * cs.inv_alpha;
                    if (fabs(pap) < 1e-30) {
                        cs.stop = STOP_BREAKDOWN; cs.xupd++; cs.final_res = sqrt(rho); cs.done = true;
                        beta = 0.0;
                    } else {
                        alpha = gamma * recip(pap);
                        cs.inv_gamma = recip(gamma);
                        cs.inv_alpha = pap * cs.inv_gamma;
                        cs.first = false;
                        cs.xupd++;
                    }
                }
                scal[3 * NR + lane] = alpha;
                scal[4 * NR + lane] = beta;
            }
            if (lane == 0) {
                ctl[0] = act;
                ctl[2] = (int)ru;
            }
            clk.lap(6);
        }
        if (a.coarse && warp > 0) {
            asm volatile("bar.sync 1, %0;" ::"r"(nt - 32) : "memory");
            coarse_apply_multi<T, NR>(Ai, a.C, rows, ct, qw, 1);
        }
        __syncthreads();
        if (ctl[3]) { status = ST_TIMEOUT; break; }
        const int act = ctl[0];
        if (act == ACT_STOP) break;
        clk.lap(5);

        if (MIXED && act == ACT_RU) {
            // ---- FP64 residuals F - K x of every case; the cases that asked
            //      replace r with it ----
            const bool mine = ((unsigned)ctl[2] >> kc) & 1u;
            for (int q = tid; q < 3 * no * NR; q += nt) {
                const int k3 = q / NR;
                Tag<double>::put(a.llx + ((size_t)(3 * gid[k3 / 3] + k3 % 3) * NR + kc) * 2, x[q], xe);
            }
            bool ok = true;
            for (int q = tid; q < 3 * nloc * NR && ok; q += nt) {
                if (q < 3 * no * NR) { xl[q] = x[q]; continue; }
                const int k3 = q / NR;
                double xv;
                ok = poll<double>(a.llx + ((size_t)(3 * gid[k3 / 3] + k3 % 3) * NR + kc) * 2, xe, xv, wt);
                xl[q] = xv;
            }
            if (__syncthreads_or(!ok)) { status = ST_TIMEOUT; break; }
            xe++;
            rows_multi64<NR>(gq, rcol, kg64, xl, ytd, no);
            __syncthreads();
            double vt[4] = {0.0, 0.0, 0.0, 0.0};
            unsigned long long* rb = a.llv + (size_t)(e & 1) * N3 * NR * 2;
            unsigned long long* qb = a.llp + (size_t)(e & 1) * kRep * a.G * SW;
            for (int q = tid; q < no * NR; q += nt) {
                const int n = q / NR, G3 = 3 * gid[n];
                double kx[3], rtv[3];
#pragma unroll
                for (int d = 0; d < 3; d++) kx[d] = ytd[(3 * n + d) * NR + kc];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const int i = (3 * n + d) * NR + kc;
                    const double rt = cm[3 * n + d] ? -xl[i] : (double)a.F[kc * N3 + G3 + d] - kx[d];
                    vt[0] += rt * rt;
                    rtv[d] = rt;
                    if (mine) r[i] = (T)rt;
                    Tag<T>::put(rb + ((size_t)(G3 + d) * NR + kc) * TW, r[i], e);
                }
                if (a.coarse) restrict3(rtv, cm + 3 * n, nb + 3 * n, vt + 1);
            }
            if (a.coarse) {
                block_publish_multi<NR, 4>(vt, red, qb, a.G, g, e);
                ok = exchange_round_multi<T, NR, 4 * NR>(qb, a.G, rb, r, no, nloc, gid, g, e, sp, wt);
            } else {
                double v1[1] = {vt[0]};
                block_publish_multi<NR, 1>(v1, red, qb, a.G, g, e);
                ok = exchange_round_multi<T, NR, NR>(qb, a.G, rb, r, no, nloc, gid, g, e, sp, wt);
            }
            if (__syncthreads_or(!ok)) { status = ST_TIMEOUT; break; }
            sum_partials<NR>(sp, a.G, a.coarse ? 4 * NR : NR, scal);
            if (a.coarse) {
                stage_coarse<T, NR>(sp, a.G, 4 * NR, NR, ct);
                __syncthreads();
                coarse_apply_multi<T, NR>(Ai, a.C, rows, ct, cvb + cb * RN, 0, (unsigned)ctl[2]);
            }
            __syncthreads();
            e++;
            // u from r for every case: the FP64 products may have used u's
            // space, and for a case that kept r and c this gives u's old bits
            for (int q = tid; q < nloc * NR; q += nt) {
                const int n = q / NR;
                T rv[3], uv[3];
#pragma unroll
                for (int d = 0; d < 3; d++) rv[d] = r[(3 * n + d) * NR + kc];
                block_jacobi3(B + 9 * n, rv, uv);
#pragma unroll
                for (int d = 0; d < 3; d++) u[(3 * n + d) * NR + kc] = uv[d];
                if (a.coarse && !cheb) {
                    const double* cv = cvb + cb * RN;
                    const int sl = 3 * nslot[n];
                    const double c3[3] = {cv[sl * NR + kc], cv[(sl + 1) * NR + kc], cv[(sl + 2) * NR + kc]};
                    prolong(n, c3);
                }
            }
            if (cheb) {
                __syncthreads();
                rows_multi<T, NR>(R, A, u, yt, nn1, a.w_rigid);
                __syncthreads();
                for (int q = tid; q < nn1 * NR; q += nt) {
                    const int n = q / NR;
                    smooth(n);
                    if (a.coarse) {
                        const double* cv = cvb + cb * RN;
                        const int sl = 3 * nslot[n];
                        const double c3[3] = {cv[sl * NR + kc], cv[(sl + 1) * NR + kc], cv[(sl + 2) * NR + kc]};
                        prolong(n, c3);
                    }
                }
            }
            __syncwarp();
            if (tid < 32) {
                const bool me = lane < NR;
                if (me && !cs.done) {
                    const double trn = sqrt(scal[lane]);
                    const int stalled = cs.xupd - cs.xupd_ref >= a.reliable_interval ? 1 : a.stall_step;
                    if (cs.asked) {
                        cs.nru++;
                        cs.rn_ref = trn;
                        cs.thr_ru = a.reliable_delta * cs.rn_ref * (a.reliable_delta * cs.rn_ref);
                        cs.xupd_ref = cs.xupd;
                    }
                    if (!isfinite(trn)) {
                        cs.status = ST_NONFINITE; cs.stop = STOP_BREAKDOWN; cs.done = true;
                    } else if ((a.stop_rule == 0 && trn < a.tol) || trn / cs.bnorm < a.tol) {
                        cs.stop = STOP_CONVERGED; cs.final_res = trn; cs.true_rel = trn / cs.bnorm; cs.done = true;
                    } else if (!cs.asked) {
                        // a replacement for another case: this one's recurrences go on
                    } else if (cs.xupd >= a.maxit) {
                        cs.stop = STOP_MAX_ITER; cs.final_res = trn; cs.true_rel = trn / cs.bnorm; cs.done = true;
                    } else if (trn < 0.5 * cs.best_trn) {
                        cs.best_trn = trn;
                        cs.stall = 0;
                    } else if ((cs.stall += stalled) >= a.stall_limit) {
                        // its own replacements without halving the FP64 residual:
                        // the FP32 inner iterations stopped helping
                        cs.stop = STOP_STAGNATED; cs.final_res = trn; cs.true_rel = trn / cs.bnorm; cs.done = true;
                    }
                }
                const unsigned dn = __ballot_sync(0xffffffffu, me && cs.done) & cmask;
                if (lane == 0) ctl[0] = dn == cmask ? ACT_STOP : ACT_UPDATE;
            }
            __syncthreads();
            if (ctl[0] == ACT_STOP) break;
            clk.lap(7);
            continue;
        }

        // ---- vector updates of every case (alpha = beta = 0 for a stopped one) ----
        const double alpha = scal[3 * NR + kc], beta = scal[4 * NR + kc];
        const T bt = (T)beta, at = (T)alpha;
        const double* cso = csb + cb * RN;
        const double* cvo = cvb + cb * RN;
        if (a.coarse)
            for (int i = tid; i < RN; i += nt) {
                const double c1 = __fma_rn(beta, cso[i], qw[i]);
                csb[(cb ^ 1) * RN + i] = c1;
                cvb[(cb ^ 1) * RN + i] = __fma_rn(-alpha, c1, cvo[i]);
            }
        auto c_new = [&](int n, double* c3) {
            const int sl = 3 * nslot[n];
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const int i = (sl + m) * NR + kc;
                c3[m] = __fma_rn(-alpha, __fma_rn(beta, cso[i], qw[i]), cvo[i]);
            }
        };
        for (int q = tid; q < nloc * NR; q += nt) {
            const int n = q / NR;
            T rv[3], uv[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const int i = (3 * n + d) * NR + kc;
                const T sk = w[i] + bt * s[i];
                s[i] = sk;
                if (cheb) {
                    if (n < no) {
                        const T pk = u[i] + bt * p[i];
                        p[i] = pk;
                        x[i] += alpha * (double)pk;
                    }
                } else {
                    const T pk = u[i] + bt * p[i];
                    p[i] = pk;
                    if (n < no) x[i] += alpha * (double)pk;
                }
                rv[d] = r[i] - at * sk;
                r[i] = rv[d];
            }
            block_jacobi3(B + 9 * n, rv, uv);
#pragma unroll
            for (int d = 0; d < 3; d++) u[(3 * n + d) * NR + kc] = uv[d];
            if (a.coarse && !cheb) {
                double c3[3];
                c_new(n, c3);
                prolong(n, c3);
            }
        }
        __syncthreads();
        clk.lap(7);
        if (cheb) {
            rows_multi<T, NR>(R, A, u, yt, nn1, a.w_rigid);
            __syncthreads();
            clk.lap(3);
            for (int q = tid; q < nn1 * NR; q += nt) {
                const int n = q / NR;
                smooth(n);
                if (a.coarse) {
                    double c3[3];
                    c_new(n, c3);
                    prolong(n, c3);
                }
            }
            __syncthreads();
            clk.lap(7);
        }
        if (a.coarse) cb ^= 1;
    }

    // ---- write x of every case; FP64 true residuals unless all known ----
    for (int q = tid; q < 3 * no * NR; q += nt) {
        const int k3 = q / NR;
        a.x[kc * N3 + 3 * gid[k3 / 3] + k3 % 3] = x[q];
    }
    if (tid < 32) {
        const unsigned need = __ballot_sync(0xffffffffu, lane < NR && cs.true_rel < 0.0) & cmask;
        if (lane == 0) ctl[1] = need ? 1 : 0;
    }
    __syncthreads();
    if (status == ST_OK && ctl[1]) {
        for (int q = tid; q < 3 * no * NR; q += nt) {
            const int k3 = q / NR;
            Tag<double>::put(a.llx + ((size_t)(3 * gid[k3 / 3] + k3 % 3) * NR + kc) * 2, x[q], xe);
        }
        bool ok = true;
        for (int q = tid; q < 3 * nloc * NR && ok; q += nt) {
            if (q < 3 * no * NR) { xl[q] = x[q]; continue; }
            const int k3 = q / NR;
            double xv;
            ok = poll<double>(a.llx + ((size_t)(3 * gid[k3 / 3] + k3 % 3) * NR + kc) * 2, xe, xv, wt);
            xl[q] = xv;
        }
        if (__syncthreads_or(!ok)) {
            status = ST_TIMEOUT;
        } else {
            if constexpr (MIXED)
                rows_multi64<NR>(gq, rcol, kg64, xl, ytd, no);
            else
                rows_multi<T, NR>(R, A, xl, ytd, no, a.w_rigid);
            __syncthreads();
            double v2[2] = {0.0, 0.0};
            for (int q = tid; q < no * NR; q += nt) {
                const int n = q / NR, G3 = 3 * gid[n];
                double kx[3];
#pragma unroll
                for (int d = 0; d < 3; d++) kx[d] = ytd[(3 * n + d) * NR + kc];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const int i = (3 * n + d) * NR + kc;
                    const double f = cm[3 * n + d] ? 0.0 : (double)a.F[kc * N3 + G3 + d];
                    const double rt = cm[3 * n + d] ? -xl[i] : f - kx[d];
                    v2[0] += rt * rt;
                    v2[1] += f * f;
                }
            }
            unsigned long long* pb = a.llp + (size_t)(e & 1) * kRep * a.G * SW;
            block_publish_multi<NR, 2>(v2, red, pb, a.G, g, e);
            if (g == 0) {
                ok = exchange_round_multi<T, NR, 2 * NR>(pb, a.G, nullptr, w, no, no, gid, g, e, sp, wt);
                if (__syncthreads_or(!ok)) {
                    status = ST_TIMEOUT;
                } else {
                    sum_partials<2 * NR>(sp, a.G, 2 * NR, scal);
                    __syncthreads();
                    if (tid < NR && cs.true_rel < 0.0)
                        cs.true_rel = scal[NR + tid] > 0 ? sqrt(scal[tid] / scal[NR + tid]) : 0.0;
                }
            }
        }
    }
    if (clk.on)
        for (int k = 0; k < 8; k++) a.res[0].phase_cycles[k] = clk.t[k];
    if (g == 0 && tid < NR) {
        PcgResult& R = a.res[tid];
        R.status = status != ST_OK ? status : cs.status;
        R.iterations = cs.xupd;
        R.converged = (cs.stop == STOP_CONVERGED || cs.stop == STOP_ZERO_RHS) ? 1 : 0;
        R.stop_reason = cs.stop < 0 ? STOP_MAX_ITER : cs.stop;
        R.final_residual = cs.final_res;
        R.true_rel_residual = cs.true_rel < 0.0 ? 0.0 : cs.true_rel;
        R.b_norm = cs.bnorm;
        R.reliable_updates = cs.nru;
        R.reductions = (int)(e - 1 - a.tag0);
        R.last_tag = e > xe ? e : xe;
    }
}

// NR load cases of one plate on the whole grid: part g = block g.  a.F and
// a.x hold NR vectors of 3 Nn back to back, a.res NR result records, and the
// exchange buffers are sized for NR cases.
template <typename T, bool MIXED, int NR>
__global__ void __launch_bounds__(kMultiThreads, 1) pcg_multi_kernel(const __grid_constant__ PcgArgs a) {
    extern __shared__ __align__(16) unsigned char sm[];
    pcg_multi_body<T, MIXED, NR>(a, blockIdx.x, sm);
}

}  // namespace pg
