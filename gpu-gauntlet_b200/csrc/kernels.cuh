// The persistent PCG kernels of the plate solver.
//
//   pcg_kernel         persistent cooperative PCG: the whole solve in one
//                      launch, one grid-wide wait per iteration
//   pcg_batch_kernel   many plates, one team of blocks per plate queue
//   (pcg_multi_kernel, several load cases of one plate in lockstep, is in
//   multi.cuh)
//
// PCG form.  The reference runs textbook PCG (pcg.ts:98-215) with three
// reductions per iteration.  Here the Chronopoulos-Gear recurrence computes
// the same iterates in exact arithmetic with one reduction per iteration:
//   w = A u;  gamma = (r,u), delta = (w,u), rho = (r,r)     [one reduction]
//   beta = gamma/gamma_prev;  alpha = gamma/(delta - beta*gamma/alpha_prev)
//   p = u + beta p;  s = w + beta s;  x += alpha p;  r -= alpha s;  u = M^-1 r
// (delta - beta*gamma/alpha_prev equals p.Ap, the reference's breakdown
// quantity).  Each thread block owns a node set; it also keeps copies of
// r, u, p, s for its ghost nodes (nodes of its elements owned elsewhere)
// and updates them with the same arithmetic as their owners, so after the
// single wait it only needs the owners' w of its ghosts -- published before
// the wait -- and no second halo exchange.
#pragma once

#include <cstdint>

#include "rows.cuh"

namespace pg {

struct PcgResult {
    int status;
    int iterations;
    int converged;
    int stop_reason;
    double final_residual;
    double true_rel_residual;
    double b_norm;
    int reliable_updates;
    int wait_failures;
    int nonfinite_it;          // reduction index where a non-finite value appeared
    int reductions;            // grid-wide reductions performed
    double nonfinite_vals[3];  // gamma, delta, rho at that reduction
    long long phase_cycles[8];  // block 0, see PhaseClock
    unsigned last_tag;         // largest round tag this launch may have written
};

// Byte offsets of the shared-memory arrays of one block (computed on the
// host from the plan's maxima; T is the inner vector type).
struct SmemLayout {
    int r, u, p, s, w, B, yt, kt;  // T (yt: the load-case kernel's row products)
    int t;                         // T: D^-1 r on every local node (Chebyshev smoother)
    int x, xl, ytd, red, scal, sp;  // double
    int qw, cs, cv;                 // double, per coarse row of the part: A_c^-1 P^T w,
                                    // A_c^-1 P^T s and c = A_c^-1 P^T r (two copies of cs, cv)
    int ctl;                        // int[4]: decision broadcast
    int dec;                        // Decision
    int clk;                        // long long[9]: phase timers
    int nb, ainv, ct;               // T: per-node basis data, A_c^-1 rows, a round's P^T w
    int nslot;                      // int
    int gid;                       // int
    int gq, go;                    // int: the row groups' q-step offsets, staged offsets
    int rcol;                      // uint16: columns of the row blocks
    int cm;                        // uint8
    int kq;                        // q-steps of row blocks the kt area holds
    int total;
};

// Copies of every block's partial sums in the exchange buffer: block g reads
// copy g mod the number of copies.  More copies mean fewer readers polling
// one line, but more stores; each block writes lines of its own (128 bytes a
// copy: with several blocks' values in one line every store meets the
// others' pollers).  Measured on the 60k-DOF plate (148 blocks, us per
// iteration): block Jacobi (the dot products only) 3.79 / 3.55 / 3.41 / 3.50 /
// 3.84 / 4.83 with 1 / 2 / 4 / 8 / 16 / 32 copies; mixed two-level Chebyshev,
// whose blocks also read 444 coarse values, 8.23 / 7.53 / 7.08 / 6.70 / 7.10 /
// 9.30.  Lines shared by 8 blocks: 3.84 and 7.74 (8 copies); coarse values in
// lines apart from the dot products': 6.88.
constexpr int kRep = 8;
__host__ __device__ constexpr int dot_copies(bool coarse) { return coarse ? kRep : 4; }

struct PcgArgs {
    int G, Nn;
    const int* node_off;
    const int* nown;
    const int* nodes;
    // row blocks (rows.cuh): group offsets of each part, q-step
    // offsets of each group, columns and blocks of each q-step
    const int* grp_off;          // [G+1]
    const int* grp_q;            // [groups+1]
    const uint16_t* rcol;        // [q-steps][30]
    const double* rk64;          // [q-steps][9][30]
    const float* rk32;
    int w_rigid;                 // 1 (Q4): a translation in w has no stiffness; see rows.cuh
    const double* binv64;        // [Nn][9]
    const float* binv32;         // [Nn][9]
    const uint8_t* cons;         // [3Nn]
    const uint8_t* shared;       // [Nn] 1: a ghost of some part
    const float* F;              // [3Nn]
    double* x;                   // [3Nn]
    unsigned long long* llv;     // [2][3Nn][2] tagged w / r values of the owners
    unsigned long long* llx;     // [3Nn][2] tagged x values (FP64 residual rounds)
    unsigned long long* llp;     // [2][kRep][G][16] tagged partial sums (kRep copies)
    int* abort_flag;
    PcgResult* res;
    double tol;
    int maxit;
    int stop_rule;
    // round tags of this launch start at tag0 + 1: the exchange buffers keep
    // older tags from earlier launches of the plan, which never match
    unsigned tag0;
    unsigned long long timeout_ns;
    int timing;
    int test_stall;  // test hook: block 0 waits once for a tag nobody writes
    // two-level preconditioner (coarse = 1): u = M_bj r + P A_c^-1 P^T r
    int coarse;
    int C;                      // coarse DOFs, 3 per part
    const int* cagg_off;        // [G+1] aggregates touching each part's nodes
    const int* node_slot;       // per part-local node: slot in its part's aggregate list
    const double* node_basis;   // per part-local node: dx, dy, 1/h
    const int* ainv_off;        // [G+1] first A_c^-1 row of each part
    const double* ainv64;       // [rows][C]
    const float* ainv32;        // [rows][C]
    int ainv_smem;
    int reliable_interval;
    // stagnated: replacements without halving the FP64 residual, one that the
    // interval brought counted once and one that the residual asked for
    // stall_step times, reach stall_limit
    int stall_limit, stall_step;
    double reliable_delta;
    // polynomial smoother (smoother = 1; needs a plan with a 2-ring halo):
    // u = a D^-1 r - b D^-1 K D^-1 r (the degree-2 Chebyshev step for
    // D^-1 K) in place of u = D^-1 r
    int smoother;
    const int* n1;                  // [G] owned + ring-1 nodes of each part
    double cheb_a, cheb_b;
    int trace_it;                   // iteration traced (-1: none)
    unsigned long long* trace;      // [G][4] globaltimer: start, published, exchanged, end
    SmemLayout L;
};

// ---------------------------------------------------------------------------
// tagged exchange between blocks (no grid barrier)
// ---------------------------------------------------------------------------
// A value a block publishes for other blocks is stored as 64-bit words
// {32-bit payload, 32-bit round tag}; an aligned 64-bit store is
// single-copy atomic, so a reader that sees the current round's tag also
// sees that round's payload -- no fence, no arrival counter, no second
// load.  FP64 values take two words (low and high halves).  Each block
// waits only for the words it needs: every block's partial sums, and its
// own ghosts' values.  Every wait has a time limit: past it the block
// raises the abort flag and the kernel ends with PG_ETIMEOUT.

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// 128-bit forms (p 16-byte aligned).  Each 64-bit half carries its own tag,
// so a reader that sees the two halves from different rounds rejects the
// pair: the pair needs no 128-bit single-copy atomicity.
__device__ __forceinline__ void ld_relaxed2(const unsigned long long* p, unsigned long long& a,
                                            unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

__device__ __forceinline__ void st_relaxed2(unsigned long long* p, unsigned long long a,
                                            unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}

template <typename T>
struct Tag;

template <>
struct Tag<float> {
    static constexpr int W = 1;
    __device__ static __forceinline__ void put(unsigned long long* p, float v, unsigned f) {
        st_relaxed(p, ((unsigned long long)f << 32) | __float_as_uint(v));
    }
    __device__ static __forceinline__ bool get(const unsigned long long* p, unsigned f, float& v) {
        const unsigned long long a = ld_relaxed(p);
        if ((unsigned)(a >> 32) != f) return false;
        v = __uint_as_float((unsigned)a);
        return true;
    }
};

template <>
struct Tag<double> {
    static constexpr int W = 2;
    __device__ static __forceinline__ void put(unsigned long long* p, double v, unsigned f) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        st_relaxed2(p, ((unsigned long long)f << 32) | (b & 0xffffffffull),
                    ((unsigned long long)f << 32) | (b >> 32));
    }
    __device__ static __forceinline__ bool get(const unsigned long long* p, unsigned f, double& v) {
        unsigned long long a, b;
        ld_relaxed2(p, a, b);
        if ((unsigned)(a >> 32) != f || (unsigned)(b >> 32) != f) return false;
        v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
        return true;
    }
};

// 1/x for the PCG scalars: the hardware's approximate reciprocal
// (rcp.approx.ftz.f64) refined by three Newton-Raphson steps
// r <- r + r (1 - x r), each of which about doubles the number of correct
// bits, so the result is within a few ulp of 1/x for normal x.  Shorter than
// a correctly rounded division on the thread-0 path every block waits on.
__device__ __forceinline__ double recip(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double e = __fma_rn(-x, r, 1.0);
        r = __fma_rn(r, e, r);
    }
    return r;
}

// Time limit of one wait (a spin loop of one thread).  The clock starts at
// the wait's first time check (after 32 failed reads), so a wait that is
// already satisfied costs no timer read.
struct Waiter {
    unsigned long long t0, limit;
    int* abort_flag;
    int* failures;
    unsigned spins;
    __device__ __forceinline__ void start(unsigned long long lim, int* ab, int* fails) {
        limit = lim;
        abort_flag = ab;
        failures = fails;
        spins = 0;
        t0 = 0;
    }
    // false when the wait must give up (time limit, or another block gave up)
    __device__ __forceinline__ bool keep_going() {
        if ((++spins & 31u) != 0) return true;
        const unsigned long long now = gtimer();
        if (spins == 32u) t0 = now;
        if (*(volatile int*)abort_flag) return false;
        if (now - t0 >= limit) {
            atomicExch(abort_flag, 1);
            atomicAdd(failures, 1);
            return false;
        }
        return true;
    }
};

template <typename T>
__device__ __forceinline__ bool poll(const unsigned long long* p, unsigned f, T& v, Waiter& wt) {
    wt.spins = 0;
    while (!Tag<T>::get(p, f, v))
        if (!wt.keep_going()) return false;
    return true;
}

// ---------------------------------------------------------------------------
// block / grid reductions (fixed order: identical bits in every block)
// ---------------------------------------------------------------------------

// Sums KM values (KM a power of two <= 32) over the 32 lanes of a warp by
// recursive halving: at each of the first log2(KM) steps a lane keeps half
// of its values and adds the partner's copy of that half (one shuffle per
// kept value), then the single remaining value is summed over the lanes
// that share it.  Lane l ends with the warp total of value l / (32 / KM):
// KM - 1 + 5 - log2(KM) shuffles instead of 5 KM.  Fixed order.
template <int KM>
__device__ __forceinline__ double warp_reduce_scatter(double (&v)[KM]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int lv = 0; (KM >> (lv + 1)) >= 1; lv++) {
        const int h = KM >> (lv + 1), o = 16 >> lv;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double keep = up ? v[h + i] : v[i];
            const double send = up ? v[i] : v[h + i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double t = v[0];
#pragma unroll
    for (int o = 16 / KM; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// Block-wide totals of the first K (<= KM) of the KM values v, published
// as this block's partial sums: copy r < kRep goes to words
// pb[r][g][2k, 2k + 1].  After the warps' own
// reduce-scatter, lane l of warp 0 adds value k = l mod KM over warps
// l / KM, l / KM + 32 / KM, ... and the 32 / KM lanes of one value finish
// with an xor butterfly: IEEE addition is commutative, so every one of them
// holds the same bits, and each writes its share of the copies.  All
// threads call it; it has one barrier, and warp 0 alone works after it, so
// `red` must not be written again before a later barrier.
template <int KM>
__device__ void block_publish(double (&v)[KM], double* red, unsigned long long* pb, int G, int g,
                              int K, unsigned f) {
    constexpr int SH = 32 / KM;  // lanes that share one value after the reduce-scatter
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double t = warp_reduce_scatter<KM>(v);
    if (lane % SH == 0) red[warp * KM + lane / SH] = t;
    __syncthreads();
    if (warp != 0) return;
    const int k = lane % KM, w0 = lane / KM;
    double tk = 0.0;
    for (int w = w0; w < nw; w += SH) tk += red[w * KM + k];
#pragma unroll
    for (int o = KM; o < 32; o <<= 1) tk += __shfl_xor_sync(0xffffffffu, tk, o);
    if (k < K)
        for (int r = w0; r < kRep; r += SH) Tag<double>::put(pb + ((size_t)r * G + g) * 16 + 2 * k, tk, f);
}

// One exchange round outside the main loop's path (the coarse start, residual
// replacements, the final residual), all threads of the block: waits for the
// K tagged FP64 partial sums of every block (staged to sp[G * K]) and for the tagged values of this block's ghost DOFs in vector
// buffer vb (written to dst[3 * no .. 3 * nloc)).  Items 0 .. ng - 1 are
// the ghosts, which their owners publish before their partial sums, then
// the partials.  Each thread takes items tid, tid + nt, tid + 2 nt, ...
// with S in flight, and refills a slot with its next item as soon as the
// slot's item has arrived: a ghost frees its slot after one round trip, so
// every partial is being polled by the time the partials come in, and the
// round costs about one L2 round trip after the last block published.
// The block that publishes last finds every other item already there; with
// S slots per thread it reads them in ceil(items / (S nt)) round trips.
// Returns false if a wait gave up.
template <typename T, int S = 3>
__device__ bool exchange_round(const unsigned long long* __restrict__ pb, int G, int K,
                               const unsigned long long* __restrict__ vb, T* dst, int no, int nloc,
                               const int* __restrict__ gid, int g, unsigned f, double* sp,
                               Waiter& wt) {
    constexpr int TW = Tag<T>::W;
    const int ng = 3 * (nloc - no), n = ng + G * K, nt = blockDim.x;
    pb += (size_t)(g % kRep) * G * 16;  // the copy of the partials part g reads
    auto addr = [&](int i) -> const unsigned long long* {
        if (i < ng) {
            const int k = 3 * no + i;
            return vb + (size_t)(3 * gid[k / 3] + k % 3) * TW;
        }
        const int q = i - ng;
        return pb + (size_t)(q / K) * 16 + 2 * (q % K);
    };
    // S slots: item index (>= n when empty) and its address
    int it[S];
    const unsigned long long* pp[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
        it[s] = threadIdx.x + s * nt;
        pp[s] = it[s] < n ? addr(it[s]) : nullptr;
    }
    int next = threadIdx.x + S * nt;
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
        if (!any) break;
        bool moved = false;
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (it[s] >= n) continue;
            if ((unsigned)(lo[s] >> 32) != f || (unsigned)(hi[s] >> 32) != f) continue;
            const int i = it[s];
            if (i >= ng) {
                sp[i - ng] = __longlong_as_double((long long)((hi[s] << 32) | (lo[s] & 0xffffffffull)));
            } else if constexpr (TW == 2) {
                dst[3 * no + i] = (T)__longlong_as_double((long long)((hi[s] << 32) | (lo[s] & 0xffffffffull)));
            } else {
                dst[3 * no + i] = (T)__uint_as_float((unsigned)lo[s]);
            }
            it[s] = next;
            next += nt;
            pp[s] = it[s] < n ? addr(it[s]) : nullptr;
            moved = true;
        }
        if (!moved && !wt.keep_going()) return false;
    }
    return true;
}

// Warp 0: adds the first K of each block's `stride` staged partials
// (sp[G][stride]) in block order (the same bits in every block) into out[K].
template <int K>
__device__ __forceinline__ void sum_partials(const double* __restrict__ sp, int G, int stride,
                                             double* out) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    double v[K];
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = 0.0;
    for (int b = lane; b < G; b += 32)
#pragma unroll
        for (int k = 0; k < K; k++) v[k] += sp[b * stride + k];
#pragma unroll
    for (int k = 0; k < K; k++)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; k++) out[k] = v[k];
}

// ---------------------------------------------------------------------------
// persistent PCG
// ---------------------------------------------------------------------------

enum { STOP_CONVERGED = 0, STOP_MAX_ITER = 1, STOP_BREAKDOWN = 2, STOP_ZERO_RHS = 3, STOP_STAGNATED = 4 };
enum { ACT_UPDATE = 0, ACT_STOP = 1, ACT_RU = 2, ACT_NONFINITE = 3, ACT_TIMEOUT = 4 };
enum { ST_OK = 0, ST_TIMEOUT = 4, ST_NONFINITE = 5 };

// Threads per block: up to kLeanThreads the build with one row group a warp
// in registers (128 registers a thread) runs, the automatic choice; above, up
// to kMaxThreads, one with none (96 registers).  The batch and load-case
// kernels always run kBatchThreads / kMultiThreads.
constexpr int kMaxThreads = 576;
constexpr int kLeanThreads = 512;
constexpr int kResident = 1;
constexpr int kBatchThreads = 512;
constexpr int kMultiThreads = 512;  // the load-case kernel (128 registers)

// Per-phase SM cycles of thread 0 of the middle block (G / 2), when timing is
// requested:
// 0 K.u, dots and publishing w, 1 unused (0), 2 block reduction and
// publishing the partials, 3 the Chebyshev smoother's K t, 4 exchange wait
// and sum of the partials, 5 the barrier after the decision, 6 warp 0's
// decision, 7 vector updates (and the residual replacement rounds of the
// mixed mode).
struct PhaseClock {
    bool on;
    long long* t;  // 8 accumulators and the last time stamp, in shared memory
    __device__ __forceinline__ void start(bool enable, long long* acc) {
        on = enable;
        t = acc;
        if (!on) return;
        for (int k = 0; k < 8; k++) t[k] = 0;
        t[8] = clock64();
    }
    __device__ __forceinline__ void lap(int k) {
        if (!on) return;
        const long long now = clock64();
        t[k] += now - t[8];
        t[8] = now;
    }
};

__device__ __forceinline__ void block_jacobi3(const float* Bn, const float* rv, float* u) {
    u[0] = Bn[0] * rv[0] + Bn[1] * rv[1] + Bn[2] * rv[2];
    u[1] = Bn[3] * rv[0] + Bn[4] * rv[1] + Bn[5] * rv[2];
    u[2] = Bn[6] * rv[0] + Bn[7] * rv[1] + Bn[8] * rv[2];
}
__device__ __forceinline__ void block_jacobi3(const double* Bn, const double* rv, double* u) {
    u[0] = Bn[0] * rv[0] + Bn[1] * rv[1] + Bn[2] * rv[2];
    u[1] = Bn[3] * rv[0] + Bn[4] * rv[1] + Bn[5] * rv[2];
    u[2] = Bn[6] * rv[0] + Bn[7] * rv[1] + Bn[8] * rv[2];
}

// Restriction of a nodal 3-vector to the node's aggregate modes (P^T v):
// mode 0 w = 1; mode 1 w = dy, thx = 1/h; mode 2 w = dx, thy = -1/h,
// constrained DOFs excluded.
template <typename V, typename T>
__device__ __forceinline__ void restrict3(const V* v, const unsigned char* c, const T* bas,
                                          double* acc) {
    const double w = c[0] ? 0.0 : (double)v[0], tx = c[1] ? 0.0 : (double)v[1];
    const double ty = c[2] ? 0.0 : (double)v[2];
    acc[0] += w;
    acc[1] += (double)bas[1] * w + (double)bas[2] * tx;
    acc[2] += (double)bas[0] * w - (double)bas[2] * ty;
}

// u += P c for one node (c = the 3 coarse values of its aggregate).
template <typename T>
__device__ __forceinline__ void prolong3(const double* cvn, const unsigned char* c, const T* bas,
                                         T* u) {
    if (!c[0]) u[0] += (T)(cvn[0] + (double)bas[1] * cvn[1] + (double)bas[0] * cvn[2]);
    if (!c[1]) u[1] += (T)((double)bas[2] * cvn[1]);
    if (!c[2]) u[2] -= (T)((double)bas[2] * cvn[2]);
}

// out[q] = sum_j Ai[q][j] y_j for the part's coarse rows q < rows; y [C] in
// shared memory, already in the rows' type (converting it here, once per row,
// cost FP32 solves more than the product: a conversion issues at an eighth of
// an FMA's rate).  Warps w0.. take two rows each, a lane columns lane,
// lane + 32, ..., so one load of y serves both rows; then FP64 sums over the
// lanes: fixed order, so every block computes the same bits for the same row.
// Bound by reading the rows from shared memory (96 KB in FP64 on the 60k-DOF
// plate, 750 cycles).
template <typename T>
__device__ __forceinline__ void coarse_apply(const T* __restrict__ Ai, int C, int rows, const T* __restrict__ y,
                                             double* __restrict__ out, int w0) {
    const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5) - w0;
    const int nw = (int)(blockDim.x >> 5) - w0;
    if (warp < 0) return;
    for (int q = 2 * warp; q < rows; q += 2 * nw) {
        const T* r0 = Ai + (size_t)q * C;
        const T* r1 = q + 1 < rows ? r0 + C : r0;
        T a0 = T(0), a1 = T(0), b0 = T(0), b1 = T(0);
        int j = lane;
#pragma unroll 4
        for (; j + 32 < C; j += 64) {
            const T y0 = y[j], y1 = y[j + 32];
            a0 = fma(r0[j], y0, a0);
            b0 = fma(r1[j], y0, b0);
            a1 = fma(r0[j + 32], y1, a1);
            b1 = fma(r1[j + 32], y1, b1);
        }
        if (j < C) {
            a0 = fma(r0[j], y[j], a0);
            b0 = fma(r1[j], y[j], b0);
        }
        const double sa = (double)a0 + (double)a1, sb = (double)b0 + (double)b1;
        // lanes below 16 go on with the first row, the others with the second
        const bool up = lane >= 16;
        double v = (up ? sb : sa) + __shfl_xor_sync(0xffffffffu, up ? sa : sb, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((lane & 15) == 0 && q + (up ? 1 : 0) < rows) out[q + (up ? 1 : 0)] = v;
    }
}

// ---------------------------------------------------------------------------
// the main loop's exchange: three warps the dot products, the others the ghosts
// ---------------------------------------------------------------------------

// One warp: the total of partial sum k over all blocks, added in a fixed
// order (lane l blocks l, l + 32, ..., then an xor butterfly, so every lane
// of every block holds the same bits).  Up to five blocks a lane are polled
// at once, straight into registers.  False if a wait gave up.
template <int SW = 16>  // words of a block's slot
__device__ __forceinline__ bool poll_total(const unsigned long long* __restrict__ pb, int G, int g, int copies, int k,
                                           unsigned f, double& out, Waiter& wt) {
    constexpr int NB = 5;
    const int lane = threadIdx.x & 31;
    pb += (size_t)(g % copies) * G * SW + 2 * k + SW * lane;
    double acc = 0.0;
    bool ok = true;
    wt.spins = 0;
    for (int base = lane; base < G && ok; base += 32 * NB, pb += 32 * SW * NB) {
        unsigned long long lo[NB], hi[NB];
        for (;;) {
            bool got = true;
#pragma unroll
            for (int i = 0; i < NB; i++) {
                lo[i] = hi[i] = (unsigned long long)f << 32;  // past the last block: 0
                if (base + 32 * i < G) ld_relaxed2(pb + 32 * SW * i, lo[i], hi[i]);
            }
#pragma unroll
            for (int i = 0; i < NB; i++) got = got && (unsigned)(lo[i] >> 32) == f && (unsigned)(hi[i] >> 32) == f;
            if (got) break;
            if (!wt.keep_going()) {
                ok = false;
                break;
            }
        }
#pragma unroll
        for (int i = 0; i < NB; i++)
            acc += __longlong_as_double((long long)((hi[i] << 32) | (lo[i] & 0xffffffffull)));
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    out = acc;
    return __all_sync(0xffffffffu, ok);
}

// Block-wide totals of the K values v of every thread, published as this
// block's partial sums: all threads store their values (red[k][thread]),
// and after one barrier warp k adds value k of all threads (lane l threads
// l, l + 32, ..., then an xor butterfly) and its first dot_copies lanes write
// one copy each.  All threads call it; `red` must not be written again before a
// later barrier.  Fewer warps than values: warp k takes values k, k + nw, ...
template <int K>
__device__ __forceinline__ void sum_publish(const double (&v)[K], double* red, unsigned long long* pb, int G, int g,
                                            unsigned f) {
    constexpr int copies = dot_copies(K > 3);
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
#pragma unroll
    for (int k = 0; k < K; k++) red[k * nt + tid] = v[k];
    __syncthreads();
    for (int k = warp; k < K; k += nw) {
        const double* q = red + k * nt + lane;
        double t = 0.0;
        if (nw == 16) {  // the automatic block size: all loads at once, a tree of additions
            double s[16];
#pragma unroll
            for (int i = 0; i < 16; i++) s[i] = q[32 * i];
#pragma unroll
            for (int h = 8; h > 0; h >>= 1)
#pragma unroll
                for (int i = 0; i < h; i++) s[i] += s[i + h];
            t = s[0];
        } else {
            for (int w = 0; w < nw; w++) t += q[32 * w];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane < copies) Tag<double>::put(pb + ((size_t)lane * G + g) * 16 + 2 * k, t, f);
    }
}

// This thread's share (items t, t + stride, ...) of the round's other
// values: the 3 (nloc - no) ghost DOFs of vector buffer vb into dst, then
// (KC = 3) partial sums 3..5 of every block into ct[3 b + m].  S items in
// flight; a slot takes its next item as soon as its item has arrived.
template <typename T, int S>
__device__ bool poll_ghosts(const unsigned long long* __restrict__ pb, int G, int KC,
                            const unsigned long long* __restrict__ vb, T* dst, int no, int nloc,
                            const int* __restrict__ gid, int g, unsigned f, T* ct, int t, int stride,
                            Waiter& wt) {
    constexpr int TW = Tag<T>::W;
    const int ng = 3 * (nloc - no), n = ng + KC * G;
    pb += (size_t)(g % kRep) * G * 16 + 6;
    auto addr = [&](int i) -> const unsigned long long* {
        if (i < ng) {
            const int k = 3 * no + i;
            return vb + (size_t)(3 * gid[k / 3] + k % 3) * TW;
        }
        return pb + (size_t)((i - ng) / 3) * 16 + 2 * ((i - ng) % 3);
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
        if (!any) break;
        bool moved = false;
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (it[s] >= n) continue;
            if ((unsigned)(lo[s] >> 32) != f || (unsigned)(hi[s] >> 32) != f) continue;
            const int i = it[s];
            if (i >= ng) {
                ct[i - ng] = (T)__longlong_as_double((long long)((hi[s] << 32) | (lo[s] & 0xffffffffull)));
            } else if constexpr (TW == 2) {
                dst[3 * no + i] = (T)__longlong_as_double((long long)((hi[s] << 32) | (lo[s] & 0xffffffffull)));
            } else {
                dst[3 * no + i] = (T)__uint_as_float((unsigned)lo[s]);
            }
            it[s] = next;
            next += stride;
            pp[s] = it[s] < n ? addr(it[s]) : nullptr;
            moved = true;
        }
        if (!moved && !wt.keep_going()) return false;
    }
    return true;
}

// One group's rows in registers: the first kRegSteps q-steps.
template <typename T>
struct RegRows {
    T k[9 * kRegSteps];
    int c[kRegSteps];  // 3 x local column
};

// Where the rows outside the registers are.
template <typename T>
struct RowMem {
    const int* gq;        // shared: [groups + 1] q-steps before each group of the part
    const int* go;        // shared: [groups] staged q-step of the group's first one, or -1
    const uint16_t* col;  // shared: [q-steps][30]
    const T* ks;          // shared: staged q-steps
    const T* kg;          // global: the part's q-steps
};

// s += q-steps [done, w) of group grp times v (lanes < 30); w0: see row_steps.
template <typename T>
__device__ __forceinline__ void rows_rest(const RowMem<T>& A, const T* __restrict__ v, int grp, int done, T w0,
                                          T (&s)[3]) {
    const int lane = threadIdx.x & 31;
    const int q0 = A.gq[grp], w = A.gq[grp + 1] - q0;
    if (done >= w || lane >= kRowLanes) return;
    const int g0 = A.go[grp];
    const uint16_t* cq = A.col + (q0 + done) * kRowLanes + lane;
    if (g0 >= 0)
        row_steps<T>(v, cq, A.ks + g0 * 9 * kRowLanes + lane, w - done, w0, s);
    else
        row_steps<T>(v, cq, A.kg + (size_t)(q0 + done) * 9 * kRowLanes + lane, w - done, w0, s);
}

// Component of K v of this lane's DOF in a group whose rows are in registers
// (w0: see row_steps).
template <typename T>
__device__ __forceinline__ T rows_reg(const RegRows<T>& R, const RowMem<T>& A, const T* __restrict__ v, int grp,
                                      bool more, T w0) {
    T s[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int q = 0; q < kRegSteps; q++) {
        const T v0 = sizeof(T) == 4 ? v[R.c[q]] - w0 : v[R.c[q]], v1 = v[R.c[q] + 1], v2 = v[R.c[q] + 2];
#pragma unroll
        for (int r = 0; r < 3; r++)
            s[r] = fma(R.k[9 * q + 3 * r + 2], v2, fma(R.k[9 * q + 3 * r + 1], v1, fma(R.k[9 * q + 3 * r], v0, s[r])));
    }
    if (more) rows_rest(A, v, grp, kRegSteps, w0, s);
    return row_join(s);
}

// ... in any other group.
template <typename T>
__device__ __forceinline__ T rows_mem(const RowMem<T>& A, const T* __restrict__ v, int grp, T w0) {
    T s[3] = {T(0), T(0), T(0)};
    rows_rest(A, v, grp, 0, w0, s);
    return row_join(s);
}

// Decision state, in shared memory and touched by warp 0 alone: registers of
// every warp are worth more than its loads.  Reciprocals of the previous
// gamma and alpha (0 before the first update, so beta = 0 and p.Ap = delta
// there) and squared thresholds keep divisions and square roots off the path
// to the barrier.
struct Decision {
    double inv_gamma, inv_alpha;
    double thr_check;         // rho at or below it needs the full tests
    double thr_abs, thr_rel, thr_ru, bnorm, best_trn, final_res, true_rel;
    int xupd, xupd_ref, nru;  // updates, at the last replacement, replacements
    int stall;                // replacements since the FP64 residual last halved (stall_step)
    int stop, first;
};

// State of one DOF (this lane's in one group of 10 nodes).
template <typename T>
struct Dof {
    T r, s, u, w;
    T b[3];  // row of the node's 3x3 inverse, cyclically from the diagonal
};

// The whole PCG solve.  T = double: plain FP64.  T = float (MIXED): inner
// iterations in FP32 with FP64 dot products, FP64 solution x, and FP64
// true-residual replacement r = F - K x ("reliable update") whenever the
// recursive residual has fallen by reliable_delta, after reliable_interval
// updates, or when it meets the tolerance (convergence is then decided on
// the true residual).
//
// Lanes and registers.  Every vector step works on groups of 10 local nodes
// (owned nodes first), one warp a group, lane 3 i + d on component d of the
// group's node i (lanes 30 and 31 idle).  Group j nw + w belongs to warp w.
// Its first NG groups (1, or 0 in the build for more threads) are resident:
// rows, vectors and block inverse in registers for the whole solve, and only
// u (or t), which the neighbours' rows read, in shared memory.  Further
// groups keep their state in shared memory.  The lanes of a row's product
// hold w of their own DOF, so dot products, the published w, the update and
// the block-Jacobi product follow in registers and shuffles.
// An iteration is bound by latency: a warp issues an instruction about every
// 7 cycles, so what counts is the number of instructions of one warp from
// barrier to barrier.  Hence one group a warp, three barriers an iteration,
// the sums over the block's threads and over the blocks one warp a value,
// and x updated behind the publication, while the block waits anyway.
// Measured (us per iteration, before: element tasks in shared memory, 16
// warps, five barriers): 60k-DOF Q4 plate on 148 blocks FP64 block Jacobi 5.13 ->
// 3.3, FP64 two-level 6.94 -> 5.82, mixed two-level Chebyshev 7.96 -> 6.68;
// 3,267-DOF plate on 9 blocks 4.18 -> 3.0; 121k-DOF DKT plate 9.38 -> 6.2.
// Two groups a warp in 8 warps (255 registers) was slower (5.7 on the 60k-DOF
// plate): one warp's instructions then make up most of the iteration.
//
// Exchange rounds: round e (e = 1, 2, ...) carries every block's partial
// sums and the owners' values of one vector (w, or the replaced r), in
// buffers [e & 1]; x rounds (for the FP64 residual) use their own tags.
// A block overwrites buffer [e & 1] only after it has seen every block's
// round e - 1 partials, and every block reads round e - 2 before it
// publishes round e - 1, so no reader can still need the old values.
template <typename T, bool MIXED, int NG, bool COARSE, bool CHEB>
__device__ __forceinline__ void pcg_body(const PcgArgs& a, const int g, unsigned char* sm) {
    constexpr int TW = Tag<T>::W;
    constexpr int NR = NG > 0 ? NG : 1;  // array bound
    const SmemLayout& L = a.L;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int n0 = a.node_off[g], nloc = a.node_off[g + 1] - n0, no = a.nown[g];
    const int nn1 = a.n1[g];
    const int gb = a.grp_off[g], ng1 = a.grp_off[g + 1] - gb;  // groups of rows (n1 of them)
    const int ngo = (no + kRowGroup - 1) / kRowGroup, ngl = (nloc + kRowGroup - 1) / kRowGroup;
    // this lane's node within a group and its DOF component
    const int li = lane / 3, ld = lane % 3;
    const bool lact = lane < kRowLanes;
    const T ca = (T)a.cheb_a, cbc = (T)a.cheb_b;
    const size_t N3 = 3 * (size_t)a.Nn;
    const int res0 = NG * nw * kRowGroup;  // nodes below res0 are resident

    // u, w, t hold every local node; r, s, B and cm the state of the nodes that
    // are not resident (index from the first of them)
    T* u = (T*)(sm + L.u);
    T* w = (T*)(sm + L.w);
    T* t = (T*)(sm + L.t);  // Chebyshev smoother: D^-1 r
    T* r = (T*)(sm + L.r) - 3 * res0;
    T* p = (T*)(sm + L.p);  // p and x: the owned nodes
    T* s = (T*)(sm + L.s) - 3 * res0;
    T* B = (T*)(sm + L.B) - 9 * res0;
    double* x = (double*)(sm + L.x);
    unsigned char* cm = (unsigned char*)(sm + L.cm) - 3 * res0;
    double* red = (double*)(sm + L.red);
    double* scal = (double*)(sm + L.scal);
    double* sp = (double*)(sm + L.sp);
    int* gid = (int*)(sm + L.gid);
    // coarse state per row of this part: c = A_c^-1 P^T r and cs = A_c^-1 P^T s
    // in two copies (copy cb is current; an update writes copy cb ^ 1, so
    // nodes can read the current copy while the new one is written), and
    // qw = A_c^-1 P^T w of the current round
    double* qw = (double*)(sm + L.qw);
    double* csb = (double*)(sm + L.cs);
    double* cvb = (double*)(sm + L.cv);
    int* ctl = (int*)(sm + L.ctl);  // [0] action, [1] final residual needed, [2] a wait gave up
    T* nb = (T*)(sm + L.nb);
    int* nslot = (int*)(sm + L.nslot);
    const int rows = COARSE ? 3 * (a.cagg_off[g + 1] - a.cagg_off[g]) : 0;
    const T* aig = COARSE ? (MIXED ? (const T*)a.ainv32 : (const T*)a.ainv64) + (size_t)a.ainv_off[g] * a.C
                            : nullptr;
    T* ais = (T*)(sm + L.ainv);
    T* ct = (T*)(sm + L.ct);  // a round's restriction P^T w (or P^T r), every aggregate
    const T* Ai = a.ainv_smem ? (const T*)ais : aig;
    // FP64 x on every local node for the true residual, in the space of w
    // (and u): neither is live then
    double* xl = (double*)(sm + L.xl);
    const T* Bg = MIXED ? (const T*)a.binv32 : (const T*)a.binv64;

    // ---- load the part ----
    int* gq = (int*)(sm + L.gq);
    int* go = (int*)(sm + L.go);
    uint16_t* rcol = (uint16_t*)(sm + L.rcol);
    T* kts = (T*)(sm + L.kt);
    const int qb = a.grp_q[gb];
    const T* kg = (MIXED ? (const T*)a.rk32 : (const T*)a.rk64) + (size_t)qb * 9 * kRowLanes;
    for (int i = tid; i <= ng1; i += nt) gq[i] = a.grp_q[gb + i] - qb;
    for (int i = tid; i < nloc; i += nt) gid[i] = a.nodes[n0 + i];
    __syncthreads();
    if (tid == 0) {
        // the q-steps not in registers go to shared memory while they fit
        int used = 0;
        for (int k = 0; k < ng1; k++) {
            const int need = max(0, gq[k + 1] - gq[k] - (k < NG * nw ? kRegSteps : 0));
            const bool fits = used + need <= L.kq;
            go[k] = fits ? used : -1;
            if (fits) used += need;
        }
        ctl[2] = 0;
    }
    for (int i = tid; i < gq[ng1] * kRowLanes; i += nt) rcol[i] = a.rcol[(size_t)qb * kRowLanes + i];
    if (COARSE) {
        for (int i = tid; i < nloc; i += nt) {
            nslot[i] = a.node_slot[n0 + i];
#pragma unroll
            for (int q = 0; q < 3; q++) nb[3 * i + q] = (T)a.node_basis[3 * (size_t)(n0 + i) + q];
        }
        for (int j = tid; j < rows; j += nt) csb[j] = 0.0;
        if (a.ainv_smem)
            for (int i = tid; i < rows * a.C; i += nt) ais[i] = aig[i];
    }
    __syncthreads();
    const RowMem<T> A{gq, go, rcol, kts, kg};
    RegRows<T> R[NR];
    unsigned more = 0;  // bit j: resident group j has q-steps beyond the registers'
    if constexpr (NG > 0) {
#pragma unroll
        for (int j = 0; j < NG; j++) {
            const int grp = warp + j * nw;
            const int w0 = grp < ng1 ? gq[grp + 1] - gq[grp] : 0;
            if (w0 > kRegSteps) more |= 1u << j;
#pragma unroll
            for (int q = 0; q < kRegSteps; q++) {
                const bool has = q < w0 && lact;
                const size_t o = has ? (size_t)(gq[grp] + q) : 0;
                R[j].c[q] = has ? 3 * (int)rcol[o * kRowLanes + lane] : 0;
#pragma unroll
                for (int k = 0; k < 9; k++) R[j].k[9 * q + k] = has ? kg[(o * 9 + k) * kRowLanes + lane] : T(0);
            }
        }
    }
    for (int k = warp; k < ng1; k += nw) {
        if (go[k] < 0) continue;
        const int skip = k < NG * nw ? kRegSteps : 0, need = gq[k + 1] - gq[k] - skip;
        const T* src = kg + (size_t)(gq[k] + skip) * 9 * kRowLanes;
        T* dst = kts + go[k] * 9 * kRowLanes;
        for (int i = lane; i < need * 9 * kRowLanes; i += 32) dst[i] = src[i];
    }
    Dof<T> D[NR];
    unsigned cbits = 0;  // bit j: this lane's DOF of resident group j is constrained
    unsigned sbits = 0;  // bit j: ... is on a node that other parts hold as a ghost
    // this DOF's row of P: its node's three coarse values enter it with m0, m1,
    // m2 (0 on constrained DOFs), and it enters their restriction likewise
    struct Prow {
        double m1, m2;
        bool m0;  // 1 or 0
        int q;    // 3 x the node's aggregate slot
    };
    auto prow = [&](int n, bool live, bool c) -> Prow {
        Prow o{0.0, 0.0, false, 0};
        if (!live) return o;
        o.q = 3 * nslot[n];
        if (c) return o;
        const T* bs = nb + 3 * n;  // dx, dy, 1/h
        if (ld == 0) {
            o.m0 = true;
            o.m1 = (double)bs[1];
            o.m2 = (double)bs[0];
        } else if (ld == 1) {
            o.m1 = (double)bs[2];
        } else {
            o.m2 = -(double)bs[2];
        }
        return o;
    };
    Prow Pr[NR];
    // start of one DOF: r = F, everything else 0
    auto load_dof = [&](int n, bool live, Dof<T>& o) -> bool {
        o = Dof<T>{};
        if (!live) return false;
        const int G3 = 3 * gid[n] + ld;
        const bool c = a.cons[G3] != 0;
        o.r = c ? T(0) : (T)a.F[G3];
#pragma unroll
        for (int q = 0; q < 3; q++) o.b[q] = Bg[(size_t)gid[n] * 9 + 3 * ld + (ld + q) % 3];
        return c;
    };
    // a group outside the registers: this lane's DOF to and from shared memory
    auto get_dof = [&](int n, bool live, Dof<T>& o) -> bool {
        o = Dof<T>{};
        if (!live) return false;
        const int k = 3 * n + ld;
        o.r = r[k];
        o.s = s[k];
        o.u = n < nn1 || !CHEB ? u[k] : T(0);
        o.w = w[k];
#pragma unroll
        for (int q = 0; q < 3; q++) o.b[q] = B[3 * k + q];
        return (cm[k] & 1) != 0;
    };
    if constexpr (NG > 0) {
#pragma unroll
        for (int j = 0; j < NG; j++) {
            const int n = (warp + j * nw) * kRowGroup + li;
            const bool c = load_dof(n, lact && n < nloc, D[j]);
            if (c) cbits |= 1u << j;
            if (lact && n < no && a.shared[gid[n]]) sbits |= 1u << j;
            Pr[j] = Prow{0.0, 0.0, false, 0};
            if (COARSE) Pr[j] = prow(n, lact && n < nloc, c);
            const T z = jacobi_lane(D[j].b, D[j].r);
            if (lact && n < nloc) (CHEB ? t : u)[3 * n + ld] = z;
            D[j].u = z;
            if (lact && n < no) {
                p[3 * n + ld] = T(0);
                x[3 * n + ld] = 0.0;
            }
        }
    }
    for (int grp = warp + NG * nw; grp < ngl; grp += nw) {
        const int n = grp * kRowGroup + li, k = 3 * n + ld;
        const bool live = lact && n < nloc;
        Dof<T> o;
        const bool c = load_dof(n, live, o);
        const T z = jacobi_lane(o.b, o.r);
        if (live) {
            cm[k] = (c ? 1 : 0) | (n < no && a.shared[gid[n]] ? 2 : 0);
            r[k] = o.r;
            s[k] = T(0);
            if (n < no) {
                p[k] = T(0);
                x[k] = 0.0;
            }
#pragma unroll
            for (int q = 0; q < 3; q++) B[3 * k + q] = o.b[q];
            (CHEB ? t : u)[k] = z;
        }
    }
    __syncthreads();

    // what an FP32 row subtracts from w (from shared memory: by a shuffle of the
    // lanes' own values, mixed solves without the smoother took 1% less, the
    // two-level Chebyshev one 1% more)
    auto own_w = [&](const T* v, int n) -> T { return MIXED && a.w_rigid && lact && n < nn1 ? v[3 * n] : T(0); };
    // runs f(n, dof, constrained, row of P, component of K v) over this warp's
    // groups below `groups`; resident ones straight from registers
    auto each_row = [&](const T* v, int groups, auto&& f) {
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int grp = warp + j * nw, n = grp * kRowGroup + li;
                if (grp < groups) f(n, D[j], ((cbits >> j) & 1u) != 0, Pr[j], rows_reg(R[j], A, v, grp, (more >> j) & 1u, own_w(v, n)));
            }
        }
        for (int grp = warp + NG * nw; grp < groups; grp += nw) {
            const int n = grp * kRowGroup + li;
            const bool live = lact && n < nloc;
            Dof<T> o;
            const bool c = get_dof(n, live, o);
            Prow pr{0.0, 0.0, false, 0};
            if (COARSE) pr = prow(n, live, c);
            f(n, o, c, pr, rows_mem(A, v, grp, own_w(v, n)));
        }
    };
    // (P c) at this lane's DOF, lane 3 i + m of a node holding value m of its
    // aggregate; all lanes of the warp call it
    auto prolong = [&](const Prow& pr, double cv) -> T {
        const int b = lane - ld;
        const double c0 = __shfl_sync(0xffffffffu, cv, b);
        const double c1 = __shfl_sync(0xffffffffu, cv, b + 1), c2 = __shfl_sync(0xffffffffu, cv, b + 2);
        return (T)fma(pr.m2, c2, fma(pr.m1, c1, pr.m0 ? c0 : 0.0));
    };
    // P^T v of this lane's DOF value added to acc[0..2]
    auto restrict_dof = [&](const Prow& pr, double v, double* acc) {
        acc[0] += pr.m0 ? v : 0.0;
        acc[1] = fma(pr.m1, v, acc[1]);
        acc[2] = fma(pr.m2, v, acc[2]);
    };
    // u = a t - b D^-1 K t (+ P c with c from cf(row of P)): the Chebyshev
    // smoother on every row, t on every local node
    auto smooth = [&](auto&& cf) {
        each_row(t, ng1, [&](int n, Dof<T>& o, bool c, const Prow& pr, T kt) {
            const bool live = lact && n < nn1;
            const T tk = live ? t[3 * n + ld] : T(0);
            T z = ca * tk - cbc * jacobi_lane(o.b, c ? tk : kt);
            if (COARSE) z += prolong(pr, cf(pr));
            if (live) u[3 * n + ld] = z;
            o.u = z;
        });
    };
    // (K x) in FP64 at this lane's DOF of group grp, x = xl, rows from memory
    auto true_row = [&](int grp) -> double {
        if constexpr (MIXED) {
            double sd[3] = {0.0, 0.0, 0.0};
            const int q0 = gq[grp];
            if (lact)
                row_steps<double>(xl, rcol + q0 * kRowLanes + lane, a.rk64 + (size_t)(qb + q0) * 9 * kRowLanes + lane,
                                  gq[grp + 1] - q0, 0.0, sd);
            return row_join(sd);
        } else {
            return rows_mem(A, (const T*)xl, grp, T(0));
        }
    };

    PhaseClock clk;
    clk.start(a.timing && g == a.G / 2 && tid == 0, (long long*)(sm + L.clk));
    Waiter wt;
    wt.start(a.timeout_ns, a.abort_flag, &a.res->wait_failures);
    unsigned e = a.tag0 + 1, xe = a.tag0 + 1;  // round tags
    int status = ST_OK;

    // ---- two-level: c0 = A_c^-1 P^T r0 (one exchange round), u0 = S r0 + P c0 ----
    if (COARSE) {
        double v0[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int n = (warp + j * nw) * kRowGroup + li;
                if (lact && n < no) restrict_dof(Pr[j], (double)D[j].r, v0);
            }
        }
        for (int grp = warp + NG * nw; grp < ngo; grp += nw) {
            const int n = grp * kRowGroup + li;
            if (lact && n < no) restrict_dof(prow(n, true, (cm[3 * n + ld] & 1) != 0), (double)r[3 * n + ld], v0);
        }
        unsigned long long* pb0 = a.llp + (size_t)(e & 1) * kRep * a.G * 16;
        block_publish<4>(v0, red, pb0, a.G, g, 3, e);
        const bool ok = exchange_round<T>(pb0, a.G, 3, nullptr, w, no, no, gid, g, e, sp, wt);
        if (__syncthreads_or(!ok)) status = ST_TIMEOUT;
        for (int i = tid; i < a.C; i += nt) ct[i] = (T)sp[i];
        __syncthreads();
        coarse_apply<T>(Ai, a.C, rows, ct, cvb, 0);
        __syncthreads();
        e++;
    }
    if (CHEB) {
        smooth([&](const Prow& pr) { return cvb[pr.q + ld]; });
        __syncthreads();
    } else if (COARSE) {
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int n = (warp + j * nw) * kRowGroup + li;
                const bool live = lact && n < nloc;
                D[j].u += prolong(Pr[j], cvb[Pr[j].q + ld]);
                if (live) u[3 * n + ld] = D[j].u;
            }
        }
        for (int grp = warp + NG * nw; grp < ngl; grp += nw) {
            const int n = grp * kRowGroup + li;
            const bool live = lact && n < nloc;
            const Prow pr = prow(n, live, live && (cm[3 * n + ld] & 1));
            const T pc = prolong(pr, cvb[pr.q + ld]);
            if (live) u[3 * n + ld] += pc;
        }
        __syncthreads();
    }

    Decision* dec = (Decision*)(sm + L.dec);
    if (tid == 0) {
        *dec = Decision{};
        dec->thr_abs = a.stop_rule == 0 ? a.tol * a.tol : 0.0;
        dec->thr_check = dec->best_trn = INFINITY;
        dec->true_rel = -1.0;
        dec->stop = -1;
        dec->first = 1;
    }
    int cb = 0;  // current copy of the coarse state
    int it = 0;

    // x += alpha p of the last update, for the resident groups: due
    // (pending) until flush()
    double alpha = 0.0;
    bool pending = false;
    auto flush = [&]() {
        if (!pending) return;
        pending = false;
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int n = (warp + j * nw) * kRowGroup + li, k = 3 * n + ld;
                if (lact && n < no) x[k] = fma(alpha, (double)p[k], x[k]);
            }
        }
    };
    // x of every local node into xl: owned ones published and copied, ghosts
    // polled; true when no wait gave up (all threads call it)
    auto share_x = [&]() -> bool {
        flush();
        __syncthreads();  // x by its other layout of threads
        for (int k = tid; k < 3 * no; k += nt) {
            Tag<double>::put(a.llx + (size_t)(3 * gid[k / 3] + k % 3) * 2, x[k], xe);
            xl[k] = x[k];
        }
        bool ok = true;
        for (int k = 3 * no + tid; k < 3 * nloc && ok; k += nt) {
            double xv = 0.0;
            ok = poll<double>(a.llx + (size_t)(3 * gid[k / 3] + k % 3) * 2, xe, xv, wt);
            xl[k] = xv;
        }
        xe++;
        return !__syncthreads_or(!ok);
    };
    // f(n, constrained, row of P, (K x)_k) over this warp's owned groups; with
    // `set` its result becomes r of the lanes' owned DOFs
    auto each_true = [&](bool set, auto&& f) {
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int grp = warp + j * nw, n = grp * kRowGroup + li;
                if (grp < ngo) {
                    double kx;
                    if constexpr (MIXED) kx = true_row(grp);
                    else kx = rows_reg(R[j], A, (const T*)xl, grp, (more >> j) & 1u, T(0));
                    const T v = f(n, ((cbits >> j) & 1u) != 0, Pr[j], kx);
                    if (set && lact && n < no) D[j].r = v;
                }
            }
        }
        for (int grp = warp + NG * nw; grp < ngo; grp += nw) {
            const int n = grp * kRowGroup + li;
            const bool own = lact && n < no, c = own && (cm[3 * n + ld] & 1);
            Prow pr{0.0, 0.0, false, 0};
            if (COARSE) pr = prow(n, own, c);
            const T v = f(n, c, pr, true_row(grp));
            if (set && own) r[3 * n + ld] = v;
        }
    };

    for (; status == ST_OK; it++) {
        const bool tr = it == a.trace_it && tid == 0;
        if (tr) a.trace[4 * g] = gtimer();
        // ---- w = A u on owned rows, BC rows, dot products, publish w ----
        double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        unsigned long long* vb = a.llv + (size_t)(e & 1) * N3 * 2;
        unsigned long long* pb = a.llp + (size_t)(e & 1) * kRep * a.G * 16;
        each_row(u, ngo, [&](int n, Dof<T>& o, bool c, const Prow& pr, T wk) {
            if (lact && n < no) {
                if (c) wk = o.u;
                o.w = wk;
                if (n >= res0) w[3 * n + ld] = wk;
                // only nodes that another part reads
                if (NG > 0 && n < res0 ? (sbits & 1u) != 0 : (cm[3 * n + ld] & 2) != 0)
                    Tag<T>::put(vb + (size_t)(3 * gid[n] + ld) * TW, wk, e);
                v[0] += (double)o.r * (double)o.u;
                v[1] += (double)wk * (double)o.u;
                v[2] += (double)o.r * (double)o.r;
                if (COARSE) restrict_dof(pr, (double)wk, v + 3);
            }
        });
        clk.lap(0);
        if (COARSE) {
            sum_publish<6>(v, red, pb, a.G, g, e);
        } else {
            const double v3[3] = {v[0], v[1], v[2]};
            sum_publish<3>(v3, red, pb, a.G, g, e);
        }
        if (tr) a.trace[4 * g + 1] = gtimer();
        clk.lap(2);
        flush();
        // ---- exchange and decision: warps 0 .. 2 the three dot products, the
        //      others the ghosts' w and the coarse partials; then warp 0 decides
        //      while the rest apply A_c^-1 to this round's P^T w ----
        const int wd = nw > 3 ? 3 : 0;  // first of the other warps (0: too few, every warp takes its share)
        if (warp >= wd) {
            const int st = nt - 32 * wd, t0 = tid - 32 * wd;
            const int items = 3 * (nloc - no) + (COARSE ? 3 * a.G : 0);
            const bool ok = items <= 2 * st
                ? poll_ghosts<T, 2>(pb, a.G, COARSE ? 3 : 0, vb, w, no, nloc, gid, g, e, ct, t0, st, wt)
                : poll_ghosts<T, 4>(pb, a.G, COARSE ? 3 : 0, vb, w, no, nloc, gid, g, e, ct, t0, st, wt);
            if (!ok) ctl[2] = 1;
        }
        double inv_g = 0.0, inv_a = 0.0, check = 0.0;
        int nupd = 0, nref = 0;
        if (warp < 3) {
            if (warp == 0) {  // the decision's state, loaded while the block waits
                inv_g = dec->inv_gamma;
                inv_a = dec->inv_alpha;
                check = dec->thr_check;
                nupd = dec->xupd;
                nref = dec->xupd_ref;
            }
            double d = 0.0;
            bool ok = true;
            for (int k = warp; k < 3; k += min(nw, 3)) {
                ok = poll_total(pb, a.G, g, dot_copies(COARSE), k, e, d, wt) && ok;
                if (lane == 0) scal[k] = d;
            }
            if (a.test_stall && it == 0 && tid == 0) {
                double never;  // a tag no block writes: the wait must run out
                ok = ok && poll<double>(a.llp + (size_t)kRep * a.G * 32, 0xffffffffu, never, wt);
            }
            if (!ok) ctl[2] = 1;
            asm volatile("bar.sync 2, %0;" ::"r"(32 * min(nw, 3)) : "memory");
        }
        if (COARSE && (warp > 0 || nw == 1)) {
            asm volatile("bar.sync 1, %0;" ::"r"(nw == 1 ? 32 : nt - 32) : "memory");
            coarse_apply<T>(Ai, a.C, rows, ct, qw, nw == 1 ? 0 : 1);
        }
        clk.lap(4);
        if (warp == 0) {
            const bool ok = ctl[2] == 0;  // the others' waits are checked behind the barrier
            const double gamma = scal[0], delta = scal[1], rho = scal[2];
            const double beta = gamma * inv_g;
            const double pap = fma(-beta * gamma, inv_a, delta);
            const double al = gamma * recip(pap);
            int act = ACT_UPDATE;
            // the common case in one test: finite sums, no stop, no
            // replacement due, no breakdown
            const double sum = fabs(gamma) + fabs(delta) + rho;
            if (!(sum < 1e300 && rho > check && fabs(pap) >= 1e-30 && nupd < a.maxit && ok) ||
                (MIXED && nupd - nref >= a.reliable_interval)) {
                if (lane == 0) {
                    int stop = -1;
                    if (!ok) {
                        act = ACT_TIMEOUT;
                    } else if (!isfinite(gamma) || !isfinite(delta) || !isfinite(rho)) {
                        if (g == 0) {
                            a.res->nonfinite_it = it;
                            a.res->nonfinite_vals[0] = gamma;
                            a.res->nonfinite_vals[1] = delta;
                            a.res->nonfinite_vals[2] = rho;
                        }
                        act = ACT_NONFINITE;
                    } else if (dec->first && rho < 1e-60) {
                        dec->bnorm = sqrt(rho);
                        dec->true_rel = 0.0;
                        stop = STOP_ZERO_RHS;
                    } else {
                        // ||r|| < tol  <=>  rho < tol^2, and so on for the other tests
                        if (dec->first) {
                            const double bn = sqrt(rho);
                            dec->bnorm = bn;
                            dec->thr_rel = a.tol * bn * (a.tol * bn);
                            dec->thr_ru = a.reliable_delta * bn * (a.reliable_delta * bn);
                            dec->thr_check = fmax(fmax(dec->thr_abs, dec->thr_rel), MIXED ? dec->thr_ru : 0.0);
                        } else {
                            const bool conv = rho < dec->thr_abs || rho < dec->thr_rel;
                            if (MIXED && (conv || rho <= dec->thr_ru || dec->xupd - dec->xupd_ref >= a.reliable_interval))
                                act = ACT_RU;
                            else if (!MIXED && conv)
                                stop = STOP_CONVERGED;
                        }
                        if (act == ACT_UPDATE && stop < 0 && dec->xupd >= a.maxit) stop = STOP_MAX_ITER;
                        if (act == ACT_UPDATE && stop < 0 && fabs(pap) < 1e-30) {
                            stop = STOP_BREAKDOWN;
                            dec->xupd++;
                        }
                    }
                    if (stop >= 0) {
                        act = ACT_STOP;
                        dec->stop = stop;
                        dec->final_res = stop == STOP_ZERO_RHS ? 0.0 : sqrt(rho);
                    }
                    ctl[1] = act == ACT_STOP && dec->true_rel < 0.0;
                }
            }
            if (lane == 0) {
                scal[3] = al;
                scal[4] = beta;
                ctl[0] = act;
            }
            clk.lap(6);
            __syncthreads();
            if (lane == 0 && act == ACT_UPDATE) {
                // off the barrier's path: the reciprocals of the next decision
                dec->first = 0;
                dec->xupd = nupd + 1;
                const double ig = recip(gamma);
                dec->inv_gamma = ig;
                dec->inv_alpha = pap * ig;
            }
        } else {
            __syncthreads();
        }
        e++;
        const int act = ctl[2] ? ACT_TIMEOUT : ctl[0];
        if (tr) a.trace[4 * g + 2] = gtimer();
        if (act == ACT_TIMEOUT) { status = ST_TIMEOUT; break; }
        if (act == ACT_NONFINITE) { status = ST_NONFINITE; break; }
        if (act == ACT_STOP) break;
        clk.lap(5);

        if (MIXED && act == ACT_RU) {
            // ---- reliable update: r = F - K x in FP64 ----
            if (!share_x()) { status = ST_TIMEOUT; break; }
            double vt[4] = {0.0, 0.0, 0.0, 0.0};
            const int KR = COARSE ? 4 : 1;
            unsigned long long* rb = a.llv + (size_t)(e & 1) * N3 * 2;
            unsigned long long* qbuf = a.llp + (size_t)(e & 1) * kRep * a.G * 16;
            each_true(true, [&](int n, bool c, const Prow& pr, double kx) -> T {
                if (!lact || n >= no) return T(0);
                const int G3 = 3 * gid[n] + ld;
                const double rt = c ? -xl[3 * n + ld] : (double)a.F[G3] - kx;
                vt[0] += rt * rt;
                Tag<T>::put(rb + (size_t)G3 * TW, (T)rt, e);
                if (COARSE) restrict_dof(pr, rt, vt + 1);
                return (T)rt;
            });
            block_publish<4>(vt, red, qbuf, a.G, g, KR, e);
            // the ghosts' r arrive in w (xl, in the same space, is dead now)
            const bool ok = exchange_round<T>(qbuf, a.G, KR, rb, w, no, nloc, gid, g, e, sp, wt);
            if (__syncthreads_or(!ok)) { status = ST_TIMEOUT; break; }
            sum_partials<1>(sp, a.G, KR, scal);
            // c = A_c^-1 P^T r from the true residual (cs is unchanged)
            if (COARSE) {
                for (int i = tid; i < a.C; i += nt) ct[i] = (T)sp[i / 3 * 4 + 1 + i % 3];
                __syncthreads();
                coarse_apply<T>(Ai, a.C, rows, ct, cvb + cb * rows, 0);
            }
            __syncthreads();
            e++;
            auto coarse_c = [&](const Prow& pr) { return cvb[cb * rows + pr.q + ld]; };
            auto restart = [&](int n, Dof<T>& o, const Prow& pr) {
                const bool live = lact && n < nloc;
                if (live && n >= no) o.r = w[3 * n + ld];
                T z = jacobi_lane(o.b, o.r);
                if (COARSE && !CHEB) z += prolong(pr, coarse_c(pr));
                if (live) (CHEB ? t : u)[3 * n + ld] = z;
                o.u = z;
            };
            if constexpr (NG > 0) {
#pragma unroll
                for (int j = 0; j < NG; j++) restart((warp + j * nw) * kRowGroup + li, D[j], Pr[j]);
            }
            for (int grp = warp + NG * nw; grp < ngl; grp += nw) {
                const int n = grp * kRowGroup + li;
                Dof<T> o;
                const bool live = lact && n < nloc, c = get_dof(n, live, o);
                Prow pr{0.0, 0.0, false, 0};
                if (COARSE && !CHEB) pr = prow(n, live, c);
                restart(n, o, pr);
                if (live) r[3 * n + ld] = o.r;
            }
            if (CHEB) {
                __syncthreads();
                smooth(coarse_c);
            }
            if (tid == 0) {
                const double trn = sqrt(scal[0]);
                int stop = -1;
                ctl[0] = ACT_UPDATE;
                ctl[1] = 0;
                dec->nru++;
                dec->thr_ru = a.reliable_delta * trn * (a.reliable_delta * trn);
                dec->thr_check = fmax(fmax(dec->thr_abs, dec->thr_rel), dec->thr_ru);
                const int stalled = dec->xupd - dec->xupd_ref >= a.reliable_interval ? 1 : a.stall_step;
                dec->xupd_ref = dec->xupd;
                if (!isfinite(trn)) {
                    ctl[0] = ACT_NONFINITE;
                } else if ((a.stop_rule == 0 && trn < a.tol) || trn / dec->bnorm < a.tol) {
                    stop = STOP_CONVERGED;
                } else if (dec->xupd >= a.maxit) {
                    stop = STOP_MAX_ITER;
                } else if (trn < 0.5 * dec->best_trn) {
                    dec->best_trn = trn;
                    dec->stall = 0;
                } else if ((dec->stall += stalled) >= a.stall_limit) {
                    // that many replacements in a row without halving the FP64
                    // residual: the FP32 inner iterations no longer reduce
                    // the error (condition number near 1 / FP32 epsilon)
                    stop = STOP_STAGNATED;
                }
                if (stop >= 0) {
                    ctl[0] = ACT_STOP;
                    dec->stop = stop;
                    dec->final_res = trn;
                    dec->true_rel = trn / dec->bnorm;
                }
            }
            __syncthreads();
            if (ctl[0] == ACT_NONFINITE) { status = ST_NONFINITE; break; }
            if (ctl[0] == ACT_STOP) break;
            clk.lap(7);
            // the next round runs on buffers [e & 1]; the other pair may still be read
            continue;
        }

        // ---- vector updates; two-level: with cs = A_c^-1 P^T s and
        //      c = A_c^-1 P^T r, P^T s = P^T w + beta P^T s and
        //      P^T r_new = P^T r - alpha P^T s give cs = qw + beta cs and
        //      c_new = c - alpha cs, so u = M_bj r_new + P c_new needs no
        //      coarse solve after the decision ----
        alpha = scal[3];
        const double beta = scal[4];
        const T bt = (T)beta, at = (T)alpha;
        const double* cso = csb + cb * rows;
        const double* cvo = cvb + cb * rows;
        for (int q = tid; q < rows; q += nt) {
            const double c1 = __fma_rn(beta, cso[q], qw[q]);
            csb[(cb ^ 1) * rows + q] = c1;
            cvb[(cb ^ 1) * rows + q] = __fma_rn(-alpha, c1, cvo[q]);
        }
        // c_new of this lane's node, value m = lane % 3 (by the recurrences)
        auto c_new = [&](const Prow& pr) -> double {
            const int q = pr.q + ld;
            return __fma_rn(-alpha, __fma_rn(beta, cso[q], qw[q]), cvo[q]);
        };
        // s, r on every local node; D^-1 r (+ P c_new) into u, or with the
        // Chebyshev smoother t = D^-1 r
        auto update = [&](int n, Dof<T>& o, const Prow& pr) {
            o.s = fma(bt, o.s, o.w);
            o.r = fma(-at, o.s, o.r);
            T z = jacobi_lane(o.b, o.r);
            if (COARSE && !CHEB) z += prolong(pr, c_new(pr));
            if (lact && n < nloc) (CHEB ? t : u)[3 * n + ld] = z;
            o.u = z;
        };
        if constexpr (NG > 0) {
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int n = (warp + j * nw) * kRowGroup + li;
                if (lact && n >= no && n < nloc) D[j].w = w[3 * n + ld];  // a ghost's w
                if (lact && n < no) p[3 * n + ld] = fma(bt, p[3 * n + ld], D[j].u);
                update(n, D[j], Pr[j]);
            }
            pending = true;
        }
        for (int grp = warp + NG * nw; grp < ngl; grp += nw) {
            const int n = grp * kRowGroup + li, k = 3 * n + ld;
            const bool live = lact && n < nloc;
            Dof<T> o;
            const bool c = get_dof(n, live, o);
            if (live && n < no) {
                const T pk = fma(bt, p[k], o.u);
                p[k] = pk;
                x[k] = fma(alpha, (double)pk, x[k]);
            }
            Prow pr{0.0, 0.0, false, 0};
            if (COARSE && !CHEB) pr = prow(n, live, c);
            update(n, o, pr);
            if (live) {
                s[k] = o.s;
                r[k] = o.r;
            }
        }
        __syncthreads();
        clk.lap(7);
        if (CHEB) {
            smooth(c_new);
            __syncthreads();
            clk.lap(3);
        }
        if (COARSE) cb ^= 1;
        if (tr) a.trace[4 * g + 3] = gtimer();
    }

    // ---- write x; FP64 true residual ||F - K x|| unless already known ----
    flush();
    __syncthreads();
    for (int k = tid; k < 3 * no; k += nt) a.x[3 * gid[k / 3] + k % 3] = x[k];
    if (status == ST_OK && ctl[1]) {
        if (!share_x()) {
            status = ST_TIMEOUT;
        } else {
            double v[2] = {0.0, 0.0};
            each_true(false, [&](int n, bool c, const Prow&, double kx) -> T {
                if (!lact || n >= no) return T(0);
                const double f = c ? 0.0 : (double)a.F[3 * gid[n] + ld];
                const double rt = c ? -xl[3 * n + ld] : f - kx;
                v[0] += rt * rt;
                v[1] += f * f;
                return T(0);
            });
            unsigned long long* pb = a.llp + (size_t)(e & 1) * kRep * a.G * 16;
            block_publish<2>(v, red, pb, a.G, g, 2, e);
            if (g == 0) {
                const bool ok = exchange_round<T>(pb, a.G, 2, nullptr, w, no, no, gid, g, e, sp, wt);
                if (__syncthreads_or(!ok)) {
                    status = ST_TIMEOUT;
                } else {
                    sum_partials<2>(sp, a.G, 2, scal);
                    __syncthreads();
                    if (tid == 0) dec->true_rel = scal[1] > 0 ? sqrt(scal[0] / scal[1]) : 0.0;
                }
            }
        }
    }
    if (clk.on)
        for (int k = 0; k < 8; k++) a.res->phase_cycles[k] = clk.t[k];
    if (g == 0 && tid == 0) {
        a.res->status = status;
        a.res->iterations = dec->xupd;
        a.res->converged = (dec->stop == STOP_CONVERGED || dec->stop == STOP_ZERO_RHS) ? 1 : 0;
        a.res->stop_reason = dec->stop < 0 ? STOP_MAX_ITER : dec->stop;
        a.res->final_residual = dec->final_res;
        a.res->true_rel_residual = dec->true_rel < 0.0 ? 0.0 : dec->true_rel;
        a.res->b_norm = dec->bnorm;
        a.res->reliable_updates = dec->nru;
        a.res->reductions = (int)(e - 1 - a.tag0);
        a.res->last_tag = e > xe ? e : xe;
    }
}

// One plate on the whole grid: part g = block g; MAXT: the launch bound.
// COARSE / CHEB: the two-level preconditioner and the Chebyshev smoother, as
// template arguments: what a method does not use takes no registers.
template <typename T, bool MIXED, int MAXT, bool COARSE, bool CHEB>
__global__ void __launch_bounds__(MAXT, 1) pcg_kernel(const __grid_constant__ PcgArgs a) {
    extern __shared__ __align__(16) unsigned char sm[];
    pcg_body<T, MIXED, MAXT <= kLeanThreads ? kResident : 0, COARSE, CHEB>(a, blockIdx.x, sm);
}

// Many independent plates in one launch.  The grid is cut into teams of consecutive blocks; teams of one size form a
// class with one queue of plates (largest estimated work first).  A free
// team takes its class's next plate: team block 0 claims a queue position
// with an atomic counter and logs it in the team's claim slot k (tag
// k + 1), where the team's other blocks read it.  Each plate is
// partitioned into as many parts as the team has blocks and has its own
// exchange buffers, so teams never wait on each other.  Team block 0
// stamps each plate's start and end (globaltimer).
struct BatchArgs {
    const PcgArgs* plates;          // [count], npe 3 or 4, one precision for all
    const int* block_team;          // [grid] team of each block
    const int* team_base;           // [teams] first block of each team
    const int* team_class;          // [teams] class of each team
    const int* class_off;           // [classes + 1] into class_queue
    const int* class_queue;         // plate ids, class by class
    const int* log_off;             // [teams + 1] each team's claim slots
    int* class_next;                // [classes] next queue position (zero at launch)
    unsigned long long* claims;     // claim slots (zero at launch)
    unsigned long long* times;      // [count][2] start / end of each plate
    int* abort_flag;
    int* claim_failures;            // waits for a claim that gave up
    unsigned long long timeout_ns;  // limit of one wait for a claim
};

template <typename T, bool MIXED, bool COARSE, bool CHEB>
__global__ void __launch_bounds__(kBatchThreads, 1) pcg_batch_kernel(const __grid_constant__ BatchArgs b) {
    extern __shared__ __align__(16) unsigned char sm[];
    volatile int* s_plate = (volatile int*)sm;  // between plates the shared memory is free
    const int g = (int)blockIdx.x - b.team_base[b.block_team[blockIdx.x]];
    for (int k = 0;; k++) {
        if (threadIdx.x == 0) {
            // the team's class queue and claim slots, re-read each time so
            // that only g and k stay live across the plate's solve
            const int team = b.block_team[blockIdx.x], cls = b.team_class[team];
            const int q0 = b.class_off[cls], qn = b.class_off[cls + 1] - q0;
            const int lo = b.log_off[team];
            unsigned pos = (unsigned)qn;  // past the end: no plate
            if (k < b.log_off[team + 1] - lo) {
                unsigned long long* slot = b.claims + lo + k;
                if (g == 0) {
                    pos = (unsigned)atomicAdd(b.class_next + cls, 1);
                    st_relaxed(slot, ((unsigned long long)(k + 1) << 32) | pos);
                } else {
                    Waiter wt;
                    wt.start(b.timeout_ns, b.abort_flag, b.claim_failures);
                    for (;;) {
                        const unsigned long long v = ld_relaxed(slot);
                        if ((unsigned)(v >> 32) == (unsigned)(k + 1)) {
                            pos = (unsigned)v;
                            break;
                        }
                        if (!wt.keep_going()) break;
                    }
                }
            }
            *s_plate = pos < (unsigned)qn ? b.class_queue[q0 + pos] : -1;
        }
        __syncthreads();
        const int pi = *s_plate;
        __syncthreads();  // read by all before the plate's data overwrite it
        if (pi < 0) break;
        // the plate's arguments, read all through the solve
        PcgArgs& a = *(PcgArgs*)sm;  // (the layouts leave the space)
        for (int i = threadIdx.x; i < (int)(sizeof(PcgArgs) / 4); i += blockDim.x)
            ((int*)&a)[i] = ((const int*)(b.plates + pi))[i];
        __syncthreads();
        if (g == 0 && threadIdx.x == 0) b.times[2 * pi] = gtimer();
        // a plate with fewer parts than the team has blocks leaves the rest idle
        if (g < a.G) {
            // with the smoother a plate on a 1-ring halo runs block Jacobi
            if (CHEB && a.smoother)
                pcg_body<T, MIXED, kResident, COARSE, CHEB>(a, g, sm);
            else
                pcg_body<T, MIXED, kResident, COARSE, false>(a, g, sm);
        }
        __syncthreads();  // shared memory is reloaded for the next plate
        if (g == 0 && threadIdx.x == 0) b.times[2 * pi + 1] = gtimer();
    }
}

}  // namespace pg
