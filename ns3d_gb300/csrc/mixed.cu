// mixed.cu -- mixed-precision solves: FP32 BiCGSTAB (FP32 vectors, FP32
// matrix copy, FP32 accumulation in the lanes) wrapped in FP64 defect
// correction.  FP64 stays on the device for the residual r = b - A x, its
// norm, the right-hand-side norm, the Krylov scalars (alpha, beta, omega,
// rho) and the solution update, so the converged solution satisfies the same
// FP64 tolerance test as the plain path (|r|^2 <= tol^2 |b|^2).
//
// One correction round of a set of systems:
//   k_dc_resid   r64 = b - A64 x (FP64), |r64|^2 (and |b|^2 in round 0);
//                last block: convergence test, scale = 1/|r64|, inner target
//   k_m32_init   f = float(r64 * scale); r = r0 = f; d = 0; p = v = 0; |f|^2
//   k_m32_loop   the BiCGSTAB iterations in FP32 on A32 d = f (one
//                persistent cooperative launch per round; small sets:
//                k_m32_chunk, mixed_chunk.cuh)
//   k_dc_step    theta minimizing |r64 - theta A64 delta|, delta = double(d) / scale
//   k_dc_update  x += theta delta
// An inner solve stops at its relative target, at the iteration budget, or
// at a breakdown (|rho| tiny, non-finite scalars); the next round restarts
// from the new FP64 residual.  iterations() reports the inner iterations.
#include <atomic>
#include <cfloat>
#include <type_traits>

#include "device.cuh"
#include "kernels.h"
#include "loop.cuh"
#include "mixed.h"

namespace ns3d {

// The six columns of a row, slots W, E, S, N, B, T, a missing one replaced by
// the row itself: from the packed table where there is one (PACKED), or from
// the table of columns.
template <bool PACKED>
__device__ __forceinline__ void row_columns(const int *nbr, const ushort4 *pack, int row, size_t np, int (&c)[6]) {
    if (PACKED && pack) {
        packed_columns(ro(pack + row), row, c);
        return;
    }
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int k = ro(nbr + d * np + row);
        c[d] = k >= 0 ? k : row;
    }
}

// FP32 row product.  A missing entry has a zero coefficient; its gather
// reads the row's own (finite) element, so all seven products are issued
// without branches (FP32 issue is plentiful on GB300).
template <bool PACKED>
__device__ __forceinline__ float spmv_f32_row(const MSys &S, int row, const float *__restrict__ x) {
    const size_t np = (size_t)S.npad;
    const float *cf = S.coef32 + row;
    int c[6];
    row_columns<PACKED>(S.nbr, S.mg.pack, row, np, c);
    float acc = ro(cf) * x[row];
    acc = __fmaf_rn(ro(cf + 1 * np), x[c[0]], acc);
    acc = __fmaf_rn(ro(cf + 3 * np), x[c[2]], acc);
    acc = __fmaf_rn(ro(cf + 5 * np), x[c[4]], acc);
    acc = __fmaf_rn(ro(cf + 6 * np), x[c[5]], acc);
    acc = __fmaf_rn(ro(cf + 4 * np), x[c[3]], acc);
    acc = __fmaf_rn(ro(cf + 2 * np), x[c[1]], acc);
    return acc;
}

// spmv_f32_row with the input vector given by a function of the column:
// the loop kernel recomputes y = D^-1 p and z = D^-1 s of neighbouring rows
// instead of waiting for their owners to store them
template <class F>
__device__ __forceinline__ float spmv_f32_fn(const MSys &S, int row, F xf) {
    const size_t np = (size_t)S.npad;
    const int *nb = S.nbr + row;
    const float *cf = S.coef32 + row;
    const int nW = nb[0 * np], nE = nb[1 * np], nS = nb[2 * np], nN = nb[3 * np], nB = nb[4 * np], nT = nb[5 * np];
    float acc = cf[0] * xf(row);
    acc = __fmaf_rn(cf[1 * np], xf(nW >= 0 ? nW : row), acc);
    acc = __fmaf_rn(cf[3 * np], xf(nS >= 0 ? nS : row), acc);
    acc = __fmaf_rn(cf[5 * np], xf(nB >= 0 ? nB : row), acc);
    acc = __fmaf_rn(cf[6 * np], xf(nT >= 0 ? nT : row), acc);
    acc = __fmaf_rn(cf[4 * np], xf(nN >= 0 ? nN : row), acc);
    acc = __fmaf_rn(cf[2 * np], xf(nE >= 0 ? nE : row), acc);
    return acc;
}

// One row of A64 x, x given by a function of the column: every operand is
// loaded before the chain of row_ordered (a missing neighbour takes the row's
// own, unused), so the loads do not wait for each other.
template <class F>
__device__ __forceinline__ double spmv_f64_fn(const MSys &S, int row, F xf) {
    const size_t np = (size_t)S.npad;
    const int *nb = S.nbr + row;
    const double *cf = S.coef64 + row;
    int col[6];
    double c[7], x[7];
#pragma unroll
    for (int d = 0; d < 6; ++d) col[d] = ro(nb + d * np);
#pragma unroll
    for (int d = 0; d < 7; ++d) c[d] = ro(cf + d * np);
    x[0] = xf(row);
#pragma unroll
    for (int d = 0; d < 6; ++d) x[d + 1] = xf(col[d] >= 0 ? col[d] : row);
    return row_ordered(row, col[0], col[1], col[2], col[3], col[4], col[5],
                       [&](double acc, int s, int) { return __fma_rn(c[s], x[s], acc); });
}
__device__ __forceinline__ double spmv_f64_row(const MSys &S, int row, const double *x) {
    return spmv_f64_fn(S, row, [&](int c) { return x[c]; });
}

// system owning global chunk c (systems in chunk order, first begins at 0;
// the last system whose first chunk is <= c, so a system without rows is
// never chosen)
template <int CAP>
__device__ __forceinline__ int msys_of_chunk(const MSetArgT<CAP> &A, int c) {
    if constexpr (CAP <= KMAX) {
        int s = 0;
#pragma unroll
        for (int q = 1; q < CAP; ++q)
            if (q < A.nsys && c >= A.sys[q].chunk_begin) s = q;
        return s;
    } else {
        int lo = 0, hi = A.nsys - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (c >= A.sys[mid].chunk_begin) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    }
}

// Flags change only between kernels (or in the last block of a system, after
// every other block of that system has passed its check), so all threads of a
// block read the same values.  `inner`: the FP32 solve must be running too.
__device__ __forceinline__ bool m_active(const MSys &S, bool inner) {
    bool act = __ldcg(&S.dc->done) == 0;
    if (inner) act = act && __ldcg(&S.st->done) == 0;
    return act;
}

#define NS3D_MCHUNK_LOOP(INNER)                                              \
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {           \
        const MSys &S = A.sys[msys_of_chunk(A, c)];                          \
        if (!m_active(S, INNER)) continue;                                    \
        const int lc = c - S.chunk_begin;

__device__ __forceinline__ bool m_arrive_last(unsigned int *counter, unsigned int total, int *sh) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int prev = atomicAdd(counter, 1u);
        sh[2] = (prev == total - 1) ? 1 : 0;
    }
    __syncthreads();
    bool last = sh[2] != 0;
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ bool finite(double x) { return isfinite(x); }

// the end of an iteration: <r0, r> and |r|^2 decide whether the inner solve
// goes on
__device__ __forceinline__ void m32_end_iteration(KState &st, double f0r, double frr) {
    st.rr = frr;
    st.iter += 1;
    st.work += 1;
    const double eps2 = (double)FLT_EPSILON * FLT_EPSILON;
    if (!finite(frr) || !finite(st.alpha) || !finite(st.w)) {
        st.done = 1;
        st.info = 1;  // breakdown: the outer round discards this correction
    } else if (!(frr > st.tol2 && st.iter < st.maxit)) {
        st.done = 1;
    } else if (fabs(f0r) < eps2 * st.r0_sqnorm || st.w == 0.0) {
        st.done = 1;  // restart needed: end the round, the next one starts afresh
    } else {
        st.beta = (f0r / st.rho) * (st.alpha / st.w);
        st.rho = f0r;
    }
}

}  // namespace ns3d
#include "mixed_chunk.cuh"
namespace ns3d {

// ---- FP64 residual and outer control -----------------------------------------
template <int CAP, int G>
__global__ void __launch_bounds__(LANES *G, 8 / G) k_dc_resid(const __grid_constant__ MSetArgT<CAP> A, int first) {
    __shared__ double sm[2 * CH + 8];  // r, b; the trees
    __shared__ int sh[4];
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    NS3D_MCHUNK_LOOP(false)
#pragma unroll
        for (int i = 0; i < RPL / G; ++i) {
            const int q = lane + (gi * (RPL / G) + i) * LANES, row = lc * CH + q;
            const double b = S.b64[row];
            const double r = b - spmv_f64_row(S, row, S.x64);
            S.r64[row] = r;
            sm[q] = r;
            sm[CH + q] = b;
        }
        __syncthreads();
        for (int j = gi; j < 2; j += G) {
            const double *v = sm + j * CH;
            const double t = lanes_tree_sum<double>(lane_dot(v, v, lane, min(CH, S.n - lc * CH)), lane,
                                                    sm + 2 * CH + 4 * j, GroupSync{gi + 1});
            if (lane == 0) S.part[2 * (size_t)lc + j] = t;
        }
        if (m_arrive_last(&S.dc->counter, (unsigned)S.nchunks, sh) && threadIdx.x < LANES) {
            double rr, bb;
            lanes_final_sum2(S.part, S.nchunks, lane, sm + 2 * CH, rr, bb, GroupSync{1});
            if (threadIdx.x == 0) {
                DCState *dc = S.dc;
                KState *st = S.st;
                dc->counter = 0;
                if (!first) dc->total_iter += st->iter;
                if (first) {
                    dc->bb = bb;
                    dc->tol2 = dc->tol * dc->tol * bb;
                }
                dc->rr = rr;
                if (first && bb == 0.0) {
                    dc->zero_rhs = 1;
                    dc->done = 1;
                    dc->total_iter = dc->maxit;
                    dc->error = dc->tol;
                    dc->info = 0;
                } else if (!finite(rr) || (!first && st->info == 1)) {
                    dc->done = 1;
                    dc->error = sqrt(rr / dc->bb);
                    dc->info = 1;  // NumericalIssue
                } else if (!(rr > dc->tol2 && dc->total_iter < dc->maxit)) {
                    dc->done = 1;
                    dc->error = sqrt(rr / dc->bb);
                    dc->info = (dc->error <= dc->tol) ? 0 : 2;
                } else {
                    dc->scale = 1.0 / sqrt(rr);
                    // reduce the normalized residual to the inner target, but
                    // not (much) further than the outer test needs
                    const double need = 0.5 * sqrt(dc->tol2 / rr);
                    dc->tin = need > dc->tin_min ? need : dc->tin_min;
                    st->done = 0;
                    st->iter = 0;
                    st->info = 0;
                    st->maxit = min(dc->inner_cap, dc->maxit - dc->total_iter);
                }
            }
        }
    }
}

// x64 = 0 for systems with a zero right-hand side (first round); the words
// that the loop with resident chunks exchanges
template <int CAP>
__global__ void k_dc_zero(const __grid_constant__ MSetArgT<CAP> A) {
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {
        const MSys &S = A.sys[msys_of_chunk(A, c)];
        const int lc = c - S.chunk_begin, r0 = lc * CH + threadIdx.x;
        if (A.resident) {
#pragma unroll
            for (int m = 0; m < RPL; ++m) S.wy[r0 + m * LANES] = S.wz[r0 + m * LANES] = 0;
            if (threadIdx.x < TAG_KINDS * MSUB)
                unit_tag_words(S)[(size_t)(threadIdx.x / MSUB) * S.nchunks * MSUB + lc * MSUB + threadIdx.x % MSUB] = 0;
            if (lc == 0 && threadIdx.x < TAG_KINDS) *tag_counter(S.part, S.nchunks, threadIdx.x) = 0;
        }
        if (!__ldcg(&S.dc->zero_rhs)) continue;
#pragma unroll
        for (int m = 0; m < RPL; ++m) S.x64[r0 + m * LANES] = 0.0;
    }
}

// ---- FP32 inner solve -------------------------------------------------------
template <int CAP, int G>
__global__ void __launch_bounds__(LANES *G, 8 / G) k_m32_init(const __grid_constant__ MSetArgT<CAP> A) {
    __shared__ float s_f[CH];
    __shared__ double sm[8];
    __shared__ int sh[4];
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    NS3D_MCHUNK_LOOP(true)
        const double scale = __ldcg(&S.dc->scale);
        double r[RPL / G];
#pragma unroll
        for (int i = 0; i < RPL / G; ++i) r[i] = S.r64[lc * CH + lane + (gi * (RPL / G) + i) * LANES];
#pragma unroll
        for (int i = 0; i < RPL / G; ++i) {
            const int q = lane + (gi * (RPL / G) + i) * LANES, row = lc * CH + q;
            const float f = (float)(r[i] * scale);
            s_f[q] = f;
            S.r[row] = f;
            S.r0[row] = f;
            S.x[row] = 0.0f;
            S.p[row] = 0.0f;
            S.v[row] = 0.0f;
        }
        __syncthreads();
        if (gi == 0) {
            float acc = 0.0f;
            const int rows = min(CH, S.n - lc * CH);
#pragma unroll
            for (int m = 0; m < RPL; ++m)
                if (lane + m * LANES < rows) acc = __fmaf_rn(s_f[lane + m * LANES], s_f[lane + m * LANES], acc);
            const double t = lanes_tree_sum<double>((double)acc, lane, sm, GroupSync{1});
            if (lane == 0) S.part[2 * (size_t)lc] = t;
        }
        if (m_arrive_last(&S.st->counter, (unsigned)S.nchunks, sh) && threadIdx.x < LANES) {
            const double bb = lanes_final_sum(S.part, S.nchunks, 2, lane, sm, GroupSync{1});
            if (threadIdx.x == 0) {
                KState *st = S.st;
                st->counter = 0;
                st->rhs_sqnorm = bb;
                st->r0_sqnorm = bb;
                st->rr = bb;
                st->tol = __ldcg(&S.dc->tin);
                st->tol2 = st->tol * st->tol * bb;
                st->rho = 1.0;
                st->alpha = 1.0;
                st->w = 1.0;
                if (!(bb > st->tol2 && 0 < st->maxit)) {
                    st->done = 1;
                } else {
                    st->beta = bb;  // (rho/1) * (1/1) with rho = <r0, r> = |r0|^2
                    st->rho = bb;
                }
            }
        }
    }
}

// ---- aggregation multilevel preconditioner (MIXED_MG) -------------------------
struct MGView {
    int n, npad;
    const int *nbr;
    const ushort4 *pack;
    const float *coef, *invdiag;
    float *x, *b, *t, *xo;  // Jacobi start, right-hand side, residual, result
};

// level k of the hierarchy of S (level 0: the FP32 system, right-hand side b0,
// Jacobi start S.p2, result x0)
__device__ __forceinline__ MGView mg_level(const MSys &S, int k, const float *b0, float *x0) {
    MGView L;
    if (k == 0) {
        L.n = S.n;
        L.npad = S.npad;
        L.nbr = S.nbr;
        L.pack = S.mg.pack;
        L.coef = S.coef32;
        L.invdiag = S.invdiag32;
        L.x = S.p2;
        L.b = const_cast<float *>(b0);
        L.t = S.t;
        L.xo = x0;
    } else {
        const MGLevel &G = S.mg.lev[k];
        L.n = G.n;
        L.npad = G.npad;
        L.nbr = G.nbr;
        L.pack = nullptr;
        L.coef = G.coef;
        L.invdiag = G.invdiag;
        L.x = G.x;
        L.b = G.b;
        L.t = G.t;
        L.xo = G.xo;
    }
    return L;
}

// row of A x at one level, x given by a function of the row (slot d+1 couples
// through neighbour d; a missing neighbour has a zero coefficient and takes
// the row itself)
template <bool PACKED, class F>
__device__ __forceinline__ float mg_spmv_fn(const MGView &L, int row, F xf) {
    const size_t np = (size_t)L.npad;
    const float *cf = L.coef + row;
    int c[6];
    if (PACKED) row_columns<PACKED>(L.nbr, L.pack, row, np, c);
    float acc = ro(cf) * xf(row);
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        if (!PACKED) {
            c[d] = ro(L.nbr + d * np + row);
            if (c[d] < 0) c[d] = row;
        }
        acc = __fmaf_rn(ro(cf + (d + 1) * np), xf(c[d]), acc);
    }
    return acc;
}
template <bool PACKED>
__device__ __forceinline__ float mg_spmv(const MGView &L, int row, const float *x) {
    return mg_spmv_fn<PACKED>(L, row, [&](int c) { return x[c]; });
}

// The passes of a V-cycle, one row each.  Down: the residual of the level's
// Jacobi start x, stored at its place among the coarse row's up to eight
// members (C.t8, so that the restriction reads 32 contiguous bytes instead of
// a member list and scattered residuals), then the restriction with the next
// level's Jacobi start.  Up: x with the coarse correction cx added on the fly
// and one damped Jacobi sweep, into xo (the neighbours still read x).
template <bool PACKED>
__device__ __forceinline__ float mg_down(const MGView &L, int r) {
    return L.b[r] - mg_spmv<PACKED>(L, r, L.x);
}
// sum over a coarse row's members in ascending order; the unused places add +0
// to a sum that starts at +0, which changes nothing
__device__ __forceinline__ float mg_sum8(const float *t8, int I) {
    const float4 a = __ldcg(reinterpret_cast<const float4 *>(t8) + 2 * I),
                 b = __ldcg(reinterpret_cast<const float4 *>(t8) + 2 * I + 1);
    float acc = 0.0f;
    for (float v : {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}) acc += v;
    return acc;
}
__device__ __forceinline__ void mg_restrict(const MGLevel &C, float w, int I) {
    const float acc = mg_sum8(C.t8, I);
    C.b[I] = acc;
    C.x[I] = w * C.invdiag[I] * acc;
}
template <bool PACKED>
__device__ __forceinline__ float mg_up(const MGView &L, const int *pos, const float *cx, float w, int r) {
    const float x = L.x[r] + cx[ro(pos + r) >> 3];
    const float t = L.b[r] - mg_spmv_fn<PACKED>(L, r, [&](int c) { return c == r ? x : L.x[c] + cx[ro(pos + c) >> 3]; });
    return x + w * L.invdiag[r] * t;
}
// store(r, value(r)) for the rows r < n of the calling thread, two at a time
// when it has that many (the loads of both in flight)
template <class Value, class Store>
__device__ __forceinline__ void mg_pass(int n, int gtid, int gth, Value value, Store store) {
    if (n <= gth) {
        if (gtid < n) store(gtid, value(gtid));
        return;
    }
    for (int r = gtid; r < n; r += 2 * gth) {
        const bool two = n - r > gth;
        const int q = two ? r + gth : r;
        const float a = value(r), b = value(q);
        store(r, a);
        if (two) store(q, b);
    }
}

// Jacobi sweeps on the coarsest level by the calling block: x = w D^-1 b,
// then `sweeps` times t = b - A x, x += w D^-1 t
__device__ void mg_coarsest(const MGView &L, float w, int sweeps) {
    for (int r = threadIdx.x; r < L.n; r += blockDim.x) L.x[r] = w * L.invdiag[r] * L.b[r];
    __syncthreads();
    for (int it = 0; it < sweeps; ++it) {
        for (int r = threadIdx.x; r < L.n; r += blockDim.x) L.t[r] = L.b[r] - mg_spmv<false>(L, r, L.x);
        __syncthreads();
        for (int r = threadIdx.x; r < L.n; r += blockDim.x) L.x[r] += w * L.invdiag[r] * L.t[r];
        __syncthreads();
    }
}

// ---- the tail of the hierarchy in shared memory ------------------------------
// The levels of a few hundred rows cost a grid barrier (1.6 us) per pass and
// next to no work, and the 30 sweeps on the coarsest one 15 us of L2 latency
// in one block while the others waited.  Every block keeps the tail's
// matrices in shared memory for the launch and runs it itself, on the same
// restricted residual and with the same arithmetic: no grid barrier inside
// the tail and none to hand out its result.
struct TailLevel {
    int n;
    float *coef, *invdiag, *x, *x2, *b, *t;  // [7][n], [n], ...
    int *nbr;                                // [6][n]
    int *agg, *mstart, *members;             // levels above the first of the tail
};
using TailLevels = TailLevel[MG_MAX + 1];

__device__ void mg_tail_load(const MGSet &G, float *mem, TailLevels &T) {
    if (threadIdx.x == 0) {
        float *q = mem;
        for (int k = G.tail; k <= G.nlev; ++k) {
            TailLevel &L = T[k];
            const int n = L.n = G.lev[k].n;
            L.coef = q;
            L.invdiag = q + 7 * n;
            L.x = q + 8 * n;
            L.x2 = q + 9 * n;
            L.b = q + 10 * n;
            L.t = q + 11 * n;
            L.nbr = reinterpret_cast<int *>(q + 12 * n);
            q += 18 * n;
            if (k > G.tail) {
                const int nf = G.lev[k - 1].n;
                L.mstart = reinterpret_cast<int *>(q);
                L.members = L.mstart + n + 1;
                L.agg = L.members + nf;
                q += n + 1 + 2 * nf;
            }
        }
    }
    __syncthreads();
    for (int k = G.tail; k <= G.nlev; ++k) {
        const MGLevel &C = G.lev[k];
        const TailLevel &L = T[k];
        for (int r = threadIdx.x; r < L.n; r += blockDim.x) {
#pragma unroll
            for (int d = 0; d < 7; ++d) L.coef[d * L.n + r] = ro(C.coef + (size_t)d * C.npad + r);
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                const int c = ro(C.nbr + (size_t)d * C.npad + r);
                L.nbr[d * L.n + r] = c >= 0 ? c : r;  // a missing neighbour takes the row itself
            }
            L.invdiag[r] = ro(C.invdiag + r);
        }
        if (k > G.tail) {
            const int nf = G.lev[k - 1].n;
            for (int r = threadIdx.x; r <= L.n; r += blockDim.x) L.mstart[r] = ro(C.mstart + r);
            for (int r = threadIdx.x; r < nf; r += blockDim.x) {
                L.members[r] = ro(C.members + r);
                L.agg[r] = ro(C.pos + r) >> 3;
            }
        }
    }
    __syncthreads();
}

template <class F>
__device__ __forceinline__ float tail_spmv(const TailLevel &L, int r, F xf) {
    float acc = L.coef[r] * xf(r);
#pragma unroll
    for (int d = 0; d < 6; ++d) acc = __fmaf_rn(L.coef[(d + 1) * L.n + r], xf(L.nbr[d * L.n + r]), acc);
    return acc;
}

// One V-cycle of the tail by the calling block, right-hand side restricted
// from the residual of the level above; returns the result.
__device__ const float *mg_tail(const MGSet &G, TailLevels &T) {
    const int K = G.nlev, tid = threadIdx.x, nth = blockDim.x;
    const float w = G.omega;
    for (int k = G.tail; k <= K; ++k) {
        const TailLevel &L = T[k];
        for (int I = tid; I < L.n; I += nth) {
            float acc = 0.0f;
            if (k == G.tail) {
                acc = mg_sum8(G.lev[k].t8, I);
            } else {
                const float *src = T[k - 1].t;
                for (int q = L.mstart[I]; q < L.mstart[I + 1]; ++q) acc += src[L.members[q]];
            }
            L.b[I] = acc;
            L.x[I] = w * L.invdiag[I] * acc;
        }
        __syncthreads();
        if (k == K) break;
        for (int r = tid; r < L.n; r += nth) L.t[r] = L.b[r] - tail_spmv(L, r, [&](int c) { return L.x[c]; });
        __syncthreads();
    }
    {
        // sweeps on the coarsest level: x and x2 in turn, one barrier per sweep
        const TailLevel &L = T[K];
        float *from = L.x, *to = L.x2;
        if (L.n <= nth) {  // one row per thread, its matrix row in registers, the warps with rows only
            const int warps = (L.n + 31) / 32;
            if (tid < 32 * warps) {
                const int r = min(tid, L.n - 1);
                float cf[7];
                int nb[6];
#pragma unroll
                for (int d = 0; d < 7; ++d) cf[d] = L.coef[d * L.n + r];
#pragma unroll
                for (int d = 0; d < 6; ++d) nb[d] = L.nbr[d * L.n + r];
                const float wd = w * L.invdiag[r], b = L.b[r];
                float x = from[r];
                for (int it = 0; it < G.sweeps; ++it) {
                    float acc = cf[0] * x;
#pragma unroll
                    for (int d = 0; d < 6; ++d) acc = __fmaf_rn(cf[d + 1], from[nb[d]], acc);
                    x += wd * (b - acc);
                    if (tid < L.n) to[r] = x;
                    float *const o = from;
                    from = to;
                    to = o;
                    asm volatile("bar.sync 9, %0;" ::"r"(32 * warps) : "memory");
                }
            }
            __syncthreads();
            from = (G.sweeps & 1) ? L.x2 : L.x;
        } else {
            for (int it = 0; it < G.sweeps; ++it) {
                for (int r = tid; r < L.n; r += nth)
                    to[r] = from[r] + w * L.invdiag[r] * (L.b[r] - tail_spmv(L, r, [&](int c) { return from[c]; }));
                __syncthreads();
                float *const o = from;
                from = to;
                to = o;
            }
        }
        if (from != L.x) {
            for (int r = tid; r < L.n; r += nth) L.x[r] = from[r];
            __syncthreads();
        }
    }
    const float *cx = T[K].x;
    for (int k = K - 1; k >= G.tail; --k) {
        const TailLevel &L = T[k];
        const int *agg = T[k + 1].agg;
        for (int r = tid; r < L.n; r += nth) {
            const float x = L.x[r] + cx[agg[r]];
            const float t = L.b[r] - tail_spmv(L, r, [&](int c) { return L.x[c] + cx[agg[c]]; });
            L.x2[r] = x + w * L.invdiag[r] * t;
        }
        __syncthreads();
        cx = L.x2;
    }
    return cx;
}

// x0 = M^-1 b0: one V-cycle -- a damped Jacobi sweep from zero, the residual
// restricted to the next level (sum over the block), ... , Jacobi sweeps on
// the coarsest level, then on the way up the correction of the coarser level
// added and one damped Jacobi sweep.  Every thread of the grid calls it (grid
// barriers between the passes); false when a barrier failed.  The fine
// level's Jacobi start x0 = w D^-1 b0 is already written by the loop phase
// that computed b0 (p or s), so the V-cycle starts with the fine residual.
// Two passes down and one up per level: the restriction writes the next
// level's Jacobi start; the way up adds the correction where x is read and
// writes its result to another vector, so it needs no barrier between the
// residual and the sweep.  (Fusing residual and restriction too, one pass per
// coarse row, measured 3-8% slower: it walks the fine rows out of order.)
// With the tail in shared memory an iteration of a 205 K-row system (five
// levels) has 21 grid barriers instead of 53 with three passes each way and
// every level in the grid: 117 -> 78 us.
template <bool PACKED>
__device__ bool mg_apply(const MSys &S, const float *b0, float *x0, TailLevels &T, GridBar *bar, unsigned int &target,
                         int *s_ok) {
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gth = gridDim.x * blockDim.x;
    // a level of at most one row per thread: warps of consecutive rows go round
    // the blocks, so that a few thousand rows do not end up on a few SMs (205 K
    // rows, five levels: 73.5 -> 72.0 ms; large levels lose 0.2% this way)
    const int spread = ((threadIdx.x / 32) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    auto first = [&](int n) { return n <= gth ? spread : gtid; };
    const int K = S.mg.nlev, tail = S.mg.tail;
    const float w = S.mg.omega;
    const float *cx = S.mg.lev[K].x;  // the coarse correction: the coarsest level's x, the other levels' xo
    for (int k = 0; k < K; ++k) {
        const MGView L = mg_level(S, k, b0, x0);
        const MGLevel &C = S.mg.lev[k + 1];
        mg_pass(L.n, first(L.n), gth, [&](int r) { return mg_down<PACKED>(L, r); },
                [&](int r, float v) { C.t8[ro(C.pos + r)] = v; });
        if (!grid_sync(bar, target, s_ok)) return false;
        if (k + 1 == tail) {
            cx = mg_tail(S.mg, T);
            break;
        }
        for (int I = first(C.n); I < C.n; I += gth) mg_restrict(C, w, I);
        if (!grid_sync(bar, target, s_ok)) return false;
    }
    if (tail > K) {
        if (blockIdx.x == 0) mg_coarsest(mg_level(S, K, b0, x0), w, S.mg.sweeps);
        if (!grid_sync(bar, target, s_ok)) return false;
    }
    for (int k = min(K, tail) - 1; k >= 0; --k) {
        const MGView L = mg_level(S, k, b0, x0);
        const int *pos = S.mg.lev[k + 1].pos;
        mg_pass(L.n, first(L.n), gth, [&](int r) { return mg_up<PACKED>(L, pos, cx, w, r); },
                [&](int r, float v) { L.xo[r] = v; });
        if (!grid_sync(bar, target, s_ok)) return false;
        cx = L.xo;
    }
    return true;
}

// the inner solve of a system runs (its outer solve is not done either)
__device__ __forceinline__ bool inner_active(const KState &k, int dc_done) { return !dc_done && !k.done; }

// Calls op(q, r) for the rows r < rows(q) of every system q with part(q):
// the systems' row ranges, concatenated in system order, are cut
// round-robin over the grid's threads (one system alone: thread t takes rows
// t, t + threads, ...).
template <int CAP, class Part, class Rows, class Op>
__device__ __forceinline__ void mg_rows(const MSetArgT<CAP> &A, Part part, Rows rows, Op op) {
    const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long gth = (long)gridDim.x * blockDim.x;
    long base = 0;
    for (int q = 0; q < A.nsys; ++q) {
        if (!part(q)) continue;
        const int n = rows(q);
        long first = gtid - base;  // smallest r >= 0 with base + r = gtid (mod gth)
        if (first < 0) first += ((-first + gth - 1) / gth) * gth;
        for (long r = first; r < n; r += gth) op(q, (int)r);
        base += n;
    }
}

// mg_apply for every system of a merged set that has a hierarchy and an
// active inner solve (which = 0: y = M^-1 p, 1: z = M^-1 s).  Pass k of the
// way down (or up) runs for the systems with more than k coarse levels, the
// coarsest sweeps of system j in block j mod gridDim.x, so every system
// takes exactly the steps and the arithmetic of mg_apply, with one set of
// grid barriers for all of them.
template <int CAP>
__device__ bool mg_apply_set(const MSetArgT<CAP> &A, const KState *sst, const int *sdc, int which, GridBar *bar,
                             unsigned int &target, int *s_ok) {
    auto on = [&](int q) { return A.sys[q].mg.nlev > 0 && inner_active(sst[q], sdc[q]); };
    auto lvl = [&](int q, int k) {
        const MSys &S = A.sys[q];
        return which == 0 ? mg_level(S, k, S.p, S.y) : mg_level(S, k, S.s, S.z);
    };
    int kmax = 0;
    for (int q = 0; q < A.nsys; ++q)
        if (on(q)) kmax = max(kmax, A.sys[q].mg.nlev);
    for (int k = 0; k < kmax; ++k) {
        auto part = [&](int q) { return on(q) && k < A.sys[q].mg.nlev; };
        mg_rows(A, part, [&](int q) { return k == 0 ? A.sys[q].n : A.sys[q].mg.lev[k].n; },
                [&](int q, int r) {
                    const MGLevel &C = A.sys[q].mg.lev[k + 1];
                    C.t8[ro(C.pos + r)] = mg_down<false>(lvl(q, k), r);
                });
        if (!grid_sync(bar, target, s_ok)) return false;
        mg_rows(A, part, [&](int q) { return A.sys[q].mg.lev[k + 1].n; },
                [&](int q, int I) { mg_restrict(A.sys[q].mg.lev[k + 1], A.sys[q].mg.omega, I); });
        if (!grid_sync(bar, target, s_ok)) return false;
    }
    {
        int j = 0;  // index of the system among those preconditioned
        for (int q = 0; q < A.nsys; ++q) {
            if (!on(q)) continue;
            if (j++ % gridDim.x != blockIdx.x) continue;
            mg_coarsest(lvl(q, A.sys[q].mg.nlev), A.sys[q].mg.omega, A.sys[q].mg.sweeps);
        }
        if (!grid_sync(bar, target, s_ok)) return false;
    }
    for (int k = kmax - 1; k >= 0; --k) {
        auto part = [&](int q) { return on(q) && k < A.sys[q].mg.nlev; };
        auto rows = [&](int q) { return k == 0 ? A.sys[q].n : A.sys[q].mg.lev[k].n; };
        mg_rows(A, part, rows, [&](int q, int r) {
            const MGLevel &C = A.sys[q].mg.lev[k + 1];
            const MGView L = lvl(q, k);
            L.xo[r] = mg_up<false>(L, C.pos, k + 1 == A.sys[q].mg.nlev ? C.x : C.xo, A.sys[q].mg.omega, r);
        });
        if (!grid_sync(bar, target, s_ok)) return false;
    }
    return true;
}

// y = M^-1 p (which = 0) or z = M^-1 s (1) for the multilevel systems of a set
template <bool PACKED, int CAP>
__device__ __forceinline__ bool mg_precondition(const MSetArgT<CAP> &A, const KState *sst, const int *sdc,
                                                int which, TailLevels &T, GridBar *bar, unsigned int &target,
                                                int *s_ok) {
    if constexpr (CAP <= KMAX) {  // one solver instance's set: a single system
        const MSys &S = A.sys[0];
        return which == 0 ? mg_apply<PACKED>(S, S.p, S.y, T, bar, target, s_ok) : mg_apply<PACKED>(S, S.s, S.z, T, bar, target, s_ok);
    } else {
        return mg_apply_set(A, sst, sdc, which, bar, target, s_ok);
    }
}

// Galerkin operator of a coarse level: per row, the sum of its block's
// diagonal and internal couplings, and per direction the couplings that
// leave the block (in the members' order).
// A block that holds a whole isolated pore cluster (no path to the inlet or
// outlet: its rows sum to zero, the block is singular) gets a coarse
// diagonal that cancels to a rounding residue; 1/residue would blow the
// coarse correction up.  Such a diagonal (below kSingular of its members'
// diagonals in magnitude) gets no coarse correction: inverse diagonal 0.
constexpr float kSingular = 1e-4f;

// Eight lanes per row, one per member: what bounds a level is the chain of
// dependent loads (members, their columns, the columns' coarse rows), which
// the lanes walk side by side; each lane then adds all members' values in
// their order.  Average launch over the levels of a 205 K-row system: 23.0 us
// with one thread per row, 7.8 us now.
__global__ void k_mg_galerkin(int npad_f, const int *__restrict__ nbr_f, const float *__restrict__ coef_f,
                              MGLevel C) {
    const unsigned int group = 0xffu << (threadIdx.x & 24);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 8 * C.n; i += gridDim.x * blockDim.x) {
        const int I = i >> 3, j = i & 7;
        const int begin = ro(C.mstart + I), count = ro(C.mstart + I + 1) - begin;
        const int m = ro(C.members + begin + min(j, count - 1));
        const float diag = coef_f[m];
        float a[6];
        unsigned int has = 0, inside = 0;
#pragma unroll
        for (int dir = 0; dir < 6; ++dir) {
            const int col = nbr_f[(size_t)dir * npad_f + m];
            a[dir] = coef_f[(size_t)(dir + 1) * npad_f + m];
            has |= (unsigned int)(col >= 0) << dir;
            inside |= (unsigned int)(col >= 0 && ro(C.pos + max(col, 0)) >> 3 == I) << dir;
        }
        float d = 0.0f, dabs = 0.0f, off[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q >= count) break;
            const float dq = __shfl_sync(group, diag, q, 8);
            const unsigned int hq = __shfl_sync(group, has, q, 8), iq = __shfl_sync(group, inside, q, 8);
            d += dq;
            dabs += fabsf(dq);
#pragma unroll
            for (int dir = 0; dir < 6; ++dir) {
                const float v = __shfl_sync(group, a[dir], q, 8);
                if (iq >> dir & 1u) d += v;
                else if (hq >> dir & 1u) off[dir] += v;
            }
        }
        float out = d;  // lane j stores slot j, lane 7 the inverse diagonal
#pragma unroll
        for (int dir = 0; dir < 6; ++dir)
            if (j == dir + 1) out = off[dir];
        if (j < 7) C.coef[(size_t)j * C.npad + I] = out;
        else C.invdiag[I] = fabsf(d) > kSingular * dabs ? 1.0f / d : 0.0f;
    }
}

// ---- the FP32 inner iterations as one persistent cooperative kernel ----------
// Same block shape, interleaving, partial regions and grid barrier as the
// FP64 loop kernel (krylov.cu), with FP32 vectors and FP32 sums inside a
// work unit (FP32 pipe), FP64 sums of the unit partials and FP64 scalars.
// FUSED: three phases and grid barriers per iteration instead of five: the
// SpMV phases recompute y = D^-1 p and z = D^-1 s at neighbouring rows from
// r, p, v (cheap in FP32) instead of waiting for a barrier after their owners
// store them; p and v alternate between two buffers so that a phase never
// overwrites what a neighbour still reads.  Otherwise the five phases of the
// FP64 loop.  Every block keeps a copy of the inner state; the kernel ends when
// every inner solve of the round is done or after `max_iters` iterations.
// All FP32 loops (also mixed_chunk.cuh) do the same arithmetic and add in the
// same order, so a system's bits do not depend on the loop that solves it.  The
// order is theirs, not the FP64 loops': the work unit is a quarter chunk
// (MUNIT = 256 rows, MRPL = 2 per lane), so a group finishes a unit in one
// round of loads, and a small system spreads over 4x more groups.

struct Pair4 {  // four elements of one or two result vectors
    float *pa, *pb;
    float4 a, b;
};
__device__ __forceinline__ float4 at4(const float *p, int i) { return reinterpret_cast<const float4 *>(p)[i]; }
template <class F>
__device__ __forceinline__ float4 each4(F f, float4 a, float4 b, float4 c) {
    return make_float4(f(a.x, b.x, c.x), f(a.y, b.y, c.y), f(a.z, b.z, c.z), f(a.w, b.w, c.w));
}

// H work units of a group, taken together so that the loads of all are in
// flight: one beyond the end (or an inactive one) falls back to rows whose
// results are then not stored.
template <int CAP, int H>
struct UnitPair {
    int si[H], lc[H];
    bool on[H];
    __device__ __forceinline__ UnitPair(const MSetArgT<CAP> &A, const KState *sst, const int *sdc, int u, int gstride,
                                        int total_units) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int v = u + h * gstride;
            on[h] = v < total_units;
            si[h] = msys_of_chunk(A, (on[h] ? v : u) / MSUB);
            lc[h] = (on[h] ? v : u) - A.sys[si[h]].chunk_begin * MSUB;
            on[h] = on[h] && inner_active(sst[si[h]], sdc[si[h]]);
        }
    }
    __device__ __forceinline__ bool none() const { return !on[0] && !on[H - 1]; }
    __device__ __forceinline__ const MSys &S(const MSetArgT<CAP> &A, int h) const { return A.sys[si[h]]; }
};

template <bool FUSED, int CAP, bool PACKED = false>
__global__ void __launch_bounds__(LOOP_THREADS, LOOP_MIN_BLOCKS)
    k_m32_loop(const __grid_constant__ MSetArgT<CAP> A, GridBar *bar, int max_iters) {
    static_assert(CAP <= LOOP_THREADS, "one thread copies each system's state");
    __shared__ KState sst[CAP];
    __shared__ int sdc[CAP];
    __shared__ double sm[LOOP_GROUPS][LANES];
    __shared__ int s_ok;
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    const GroupSync gsync{gi + 1};
    const int gstride = gridDim.x * LOOP_GROUPS;
    const int cbegin = blockIdx.x + gridDim.x * gi;
    const int total_units = A.total_chunks * MSUB;
    if (threadIdx.x < A.nsys) {
        sst[threadIdx.x] = *A.sys[threadIdx.x].st;
        sdc[threadIdx.x] = A.sys[threadIdx.x].dc->done;
    }
    extern __shared__ float tail_mem[];  // the tail of a single system's hierarchy (mg_tail_words)
    __shared__ TailLevels s_tail;
    if constexpr (!FUSED && CAP <= KMAX)
        if (A.sys[0].mg.nlev > 0 && A.sys[0].mg.tail <= A.sys[0].mg.nlev) mg_tail_load(A.sys[0].mg, tail_mem, s_tail);
    unsigned int target = grid_sync_start(bar);
    __syncthreads();
    __shared__ double s_sum[CAP][2];
    // two reductions (pairs at 2 n x of the partials) of every active system
    // into s_sum, one group each
    auto two_sums = [&](int region) {
#pragma unroll 1
        for (int task = gi; task < 2 * A.nsys; task += LOOP_GROUPS) {
            const int q = task >> 1, j = task & 1;
            if (!inner_active(sst[q], sdc[q])) continue;
            const MSys &S = A.sys[q];
            const double t = lanes_final_sum<16>(S.part + region * (size_t)S.nchunks * MSUB + j, S.nchunks * MSUB, 2, lane,
                                                 sm[gi], gsync);
            if (lane == 0) s_sum[q][j] = t;
        }
        __syncthreads();
    };
    // A walk over whole chunks: op(system index, system, i) for the chunks of
    // the systems with on(system index), which takes elements 4 i .. 4 i + 3
    // and 4 (i + LANES) .. 4 (i + LANES) + 3.  An element belongs to the same
    // thread in every such walk.
    auto each_chunk = [&](auto on, auto op) {
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = msys_of_chunk(A, c);
            if (!on(si)) continue;
            const MSys &S = A.sys[si];
            op(si, S, (c - S.chunk_begin) * (CH / 4) + lane);
        }
    };
    // An element-wise phase: op(system index, system, i) computes elements
    // 4 i .. 4 i + 3 of one or two result vectors.  A group takes whole chunks,
    // a lane two float4 of each vector at once: with one row in flight per
    // thread K1, K3 and K5 took 30, 28 and 58 us at 3.6 M rows, now 11, 9 and 32.
    auto stream_chunks = [&](auto op) {
        each_chunk([&](int si) { return inner_active(sst[si], sdc[si]); }, [&](int si, const MSys &S, int i) {
            const Pair4 e0 = op(si, S, i), e1 = op(si, S, i + LANES);
            reinterpret_cast<float4 *>(e0.pa)[i] = e0.a;
            if (e0.pb) reinterpret_cast<float4 *>(e0.pb)[i] = e0.b;
            reinterpret_cast<float4 *>(e1.pa)[i + LANES] = e1.a;
            if (e1.pb) reinterpret_cast<float4 *>(e1.pb)[i + LANES] = e1.b;
        });
    };
    static_assert(CH == 8 * LANES, "two float4 a lane");
    {  // a launch that finds every system done returns at once
        bool any = false;
        for (int q = 0; q < A.nsys; ++q) any = any || inner_active(sst[q], sdc[q]);
        if (!any) max_iters = 0;
    }
    // a phase over work units, two at a time when a group has that many
    auto unit_phase = [&](auto run) {
        if (total_units > gstride) run(std::integral_constant<int, 2>());
        else run(std::integral_constant<int, 1>());
    };
    int it = 0;
    for (; it < max_iters; ++it) {
        if constexpr (FUSED) {
            const bool odd = (it & 1) != 0;
            // A: p' = r + beta (p - w v), y = D^-1 p' (stored for the own rows,
            //    recomputed for neighbours); v' = A y, <r0, v'>.  p and v are read
            //    from one buffer and written to the other.
            for (int u = cbegin; u < total_units; u += gstride) {
                const int si = msys_of_chunk(A, u / MSUB);
                if (!inner_active(sst[si], sdc[si])) continue;
                const MSys &S = A.sys[si];
                const int lc = u - S.chunk_begin * MSUB;
                const int r0 = lc * MUNIT + lane;
                const float beta = (float)sst[si].beta, w = (float)sst[si].w;
                const float *pc = odd ? S.p2 : S.p, *vc = odd ? S.v2 : S.v;
                float *pn = odd ? S.p : S.p2, *vn = odd ? S.v : S.v2;
                auto yf = [&](int k) { return S.invdiag32[k] * __fmaf_rn(beta, __fmaf_rn(-w, vc[k], pc[k]), S.r[k]); };
                float a = 0.0f;
    #pragma unroll
                for (int m = 0; m < MRPL; ++m) {
                    const int row = r0 + m * LANES;
                    const float p = __fmaf_rn(beta, __fmaf_rn(-w, vc[row], pc[row]), S.r[row]);
                    pn[row] = p;
                    S.y[row] = S.invdiag32[row] * p;
                    const float v = spmv_f32_fn(S, row, yf);
                    vn[row] = v;
                    if (row < S.n) a = __fmaf_rn(S.r0[row], v, a);
                }
                const float t = lanes_tree_sum<float>(a, lane, reinterpret_cast<float *>(sm[gi]), gsync);
                if (lane == 0) S.part[4 * (size_t)S.nchunks * MSUB + lc] = (double)t;
            }
            if (!grid_sync(bar, target, &s_ok)) break;
            for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
                if (!inner_active(sst[q], sdc[q])) continue;
                const MSys &S = A.sys[q];
                const double d = lanes_final_sum(S.part + 4 * (size_t)S.nchunks * MSUB, S.nchunks * MSUB, 1, lane, sm[gi], gsync);
                if (lane == 0) sst[q].alpha = sst[q].rho / d;
            }
            __syncthreads();
            // B: s = r - alpha v', z = D^-1 s (stored for the own rows, recomputed
            //    for neighbours); t = A z, <t, t>, <t, s>
            for (int u = cbegin; u < total_units; u += gstride) {
                const int si = msys_of_chunk(A, u / MSUB);
                if (!inner_active(sst[si], sdc[si])) continue;
                const MSys &S = A.sys[si];
                const int lc = u - S.chunk_begin * MSUB;
                const int r0 = lc * MUNIT + lane;
                const float alpha = (float)sst[si].alpha;
                const float *vn = odd ? S.v : S.v2;
                auto zf = [&](int k) { return S.invdiag32[k] * __fmaf_rn(-alpha, vn[k], S.r[k]); };
                float att = 0.0f, ats = 0.0f;
    #pragma unroll
                for (int m = 0; m < MRPL; ++m) {
                    const int row = r0 + m * LANES;
                    const float sv = __fmaf_rn(-alpha, vn[row], S.r[row]);
                    S.s[row] = sv;
                    S.z[row] = S.invdiag32[row] * sv;
                    const float t = spmv_f32_fn(S, row, zf);
                    S.t[row] = t;
                    if (row < S.n) {
                        att = __fmaf_rn(t, t, att);
                        ats = __fmaf_rn(t, sv, ats);
                    }
                }
                float tt, ts;
                lanes_tree_sum2<float>(att, ats, lane, reinterpret_cast<float *>(sm[gi]), tt, ts, gsync);
                if (lane == 0) reinterpret_cast<double2 *>(S.part)[lc] = make_double2(tt, ts);
            }
            if (!grid_sync(bar, target, &s_ok)) break;
            for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
                if (!inner_active(sst[q], sdc[q])) continue;
                const MSys &S = A.sys[q];
                double ftt, fts;
                lanes_final_sum2(S.part, S.nchunks * MSUB, lane, sm[gi], ftt, fts, gsync);
                if (lane == 0) sst[q].w = (ftt > 0.0) ? fts / ftt : 0.0;
            }
            __syncthreads();
            // C: x += alpha y + w z; r = s - w t; <r0, r>, <r, r>
            for (int u = cbegin; u < total_units; u += gstride) {
                const int si = msys_of_chunk(A, u / MSUB);
                if (!inner_active(sst[si], sdc[si])) continue;
                const MSys &S = A.sys[si];
                const int lc = u - S.chunk_begin * MSUB;
                const int r0 = lc * MUNIT + lane;
                const float alpha = (float)sst[si].alpha, w = (float)sst[si].w;
                float a0r = 0.0f, arr = 0.0f;
    #pragma unroll
                for (int m = 0; m < MRPL; ++m) {
                    const int row = r0 + m * LANES;
                    S.x[row] = __fmaf_rn(w, S.z[row], __fmaf_rn(alpha, S.y[row], S.x[row]));
                    const float r = __fmaf_rn(-w, S.t[row], S.s[row]);
                    S.r[row] = r;
                    if (row < S.n) {
                        a0r = __fmaf_rn(S.r0[row], r, a0r);
                        arr = __fmaf_rn(r, r, arr);
                    }
                }
                float t0r, trr;
                lanes_tree_sum2<float>(a0r, arr, lane, reinterpret_cast<float *>(sm[gi]), t0r, trr, gsync);
                if (lane == 0)
                    reinterpret_cast<double2 *>(S.part + 2 * (size_t)S.nchunks * MSUB)[lc] = make_double2(t0r, trr);
            }
            if (!grid_sync(bar, target, &s_ok)) break;
            for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
                if (!inner_active(sst[q], sdc[q])) continue;
                const MSys &S = A.sys[q];
                double f0r, frr;
                lanes_final_sum2(S.part + 2 * (size_t)S.nchunks * MSUB, S.nchunks * MSUB, lane, sm[gi], f0r, frr, gsync);
                if (lane == 0) m32_end_iteration(sst[q], f0r, frr);
            }
            __syncthreads();
        } else {
            // the preconditioner is multilevel for a single-system set with a
            // hierarchy (uniform across the grid: the scalars are per-block copies)
            bool mg_on = false;
            if constexpr (CAP <= KMAX) {
                mg_on = A.nsys == 1 && A.sys[0].mg.nlev > 0 && inner_active(sst[0], sdc[0]);
            } else {
                for (int q = 0; q < A.nsys; ++q)
                    mg_on = mg_on || (A.sys[q].mg.nlev > 0 && inner_active(sst[q], sdc[q]));
            }
            // p = r + beta (p - w v); y = D^-1 p
            stream_chunks([&](int si, const MSys &S, int i) {
                const float beta = (float)sst[si].beta, w = (float)sst[si].w;
                float4 p = at4(S.p, i);
                const float4 v = at4(S.v, i), r = at4(S.r, i), d = at4(S.invdiag32, i);
                // a system with a hierarchy: the V-cycle's start w D^-1 p
                float *const out = S.mg.nlev > 0 ? S.p2 : S.y;
                const float om = S.mg.omega;
                const bool mg = S.mg.nlev > 0;
                p = each4([&](float p1, float v1, float r1) { return __fmaf_rn(beta, __fmaf_rn(-w, v1, p1), r1); }, p, v, r);
                const float4 y = each4([&](float d1, float p1, float) { return mg ? om * d1 * p1 : d1 * p1; }, d, p, p);
                return Pair4{S.p, out, p, y};
            });
            if (!grid_sync(bar, target, &s_ok)) break;
            // multilevel preconditioning: y = M^-1 p (replaces the Jacobi y)
            if (mg_on && !mg_precondition<PACKED>(A, sst, sdc, 0, s_tail, bar, target, &s_ok)) break;
            // v = A y, <r0, v>
            unit_phase([&](auto units) {
                constexpr int H = decltype(units)::value;
                for (int u = cbegin; u < total_units; u += H * gstride) {
                    const UnitPair<CAP, H> U(A, sst, sdc, u, gstride, total_units);
                    if (U.none()) continue;
                    float v[H][MRPL], q[H][MRPL], a[2] = {0.0f, 0.0f};
#pragma unroll
                    for (int h = 0; h < H; ++h)
#pragma unroll
                        for (int m = 0; m < MRPL; ++m) {
                            const int row = U.lc[h] * MUNIT + lane + m * LANES;
                            v[h][m] = spmv_f32_row<PACKED>(U.S(A, h), row, U.S(A, h).y);
                            q[h][m] = U.S(A, h).r0[row];
                        }
#pragma unroll
                    for (int h = 0; h < H; ++h)
                        if (U.on[h])
#pragma unroll
                            for (int m = 0; m < MRPL; ++m) {
                                const int row = U.lc[h] * MUNIT + lane + m * LANES;
                                U.S(A, h).v[row] = v[h][m];
                                if (row < U.S(A, h).n) a[h] = __fmaf_rn(q[h][m], v[h][m], a[h]);
                            }
                    float t[2];
                    lanes_tree_sum2<float>(a[0], a[1], lane, reinterpret_cast<float *>(sm[gi]), t[0], t[1], gsync);
                    if (lane == 0)
#pragma unroll
                        for (int h = 0; h < H; ++h)
                            if (U.on[h]) U.S(A, h).part[4 * (size_t)U.S(A, h).nchunks * MSUB + U.lc[h]] = (double)t[h];
                }
            });
            if (!grid_sync(bar, target, &s_ok)) break;
            for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
                if (!inner_active(sst[q], sdc[q])) continue;
                const MSys &S = A.sys[q];
                const double d = lanes_final_sum<16>(S.part + 4 * (size_t)S.nchunks * MSUB, S.nchunks * MSUB, 1, lane, sm[gi], gsync);
                if (lane == 0) sst[q].alpha = sst[q].rho / d;
            }
            __syncthreads();
            // s = r - alpha v; z = D^-1 s
            stream_chunks([&](int si, const MSys &S, int i) {
                const float alpha = (float)sst[si].alpha;
                const float4 v = at4(S.v, i), r = at4(S.r, i), d = at4(S.invdiag32, i);
                float *const out = S.mg.nlev > 0 ? S.p2 : S.z;
                const float om = S.mg.omega;
                const bool mg = S.mg.nlev > 0;
                const float4 sv = each4([&](float v1, float r1, float) { return __fmaf_rn(-alpha, v1, r1); }, v, r, r);
                const float4 z = each4([&](float d1, float s1, float) { return mg ? om * d1 * s1 : d1 * s1; }, d, sv, sv);
                return Pair4{S.s, out, sv, z};
            });
            if (!grid_sync(bar, target, &s_ok)) break;
            if (mg_on && !mg_precondition<PACKED>(A, sst, sdc, 1, s_tail, bar, target, &s_ok)) break;
            // t = A z, <t, t>, <t, s>
            unit_phase([&](auto units) {
                constexpr int H = decltype(units)::value;
                for (int u = cbegin; u < total_units; u += H * gstride) {
                    const UnitPair<CAP, H> U(A, sst, sdc, u, gstride, total_units);
                    if (U.none()) continue;
                    float t[H][MRPL], q[H][MRPL], att[H] = {}, ats[H] = {};
#pragma unroll
                    for (int h = 0; h < H; ++h)
#pragma unroll
                        for (int m = 0; m < MRPL; ++m) {
                            const int row = U.lc[h] * MUNIT + lane + m * LANES;
                            t[h][m] = spmv_f32_row<PACKED>(U.S(A, h), row, U.S(A, h).z);
                            q[h][m] = U.S(A, h).s[row];
                        }
#pragma unroll
                    for (int h = 0; h < H; ++h)
                        if (U.on[h])
#pragma unroll
                            for (int m = 0; m < MRPL; ++m) {
                                const int row = U.lc[h] * MUNIT + lane + m * LANES;
                                U.S(A, h).t[row] = t[h][m];
                                if (row < U.S(A, h).n) {
                                    att[h] = __fmaf_rn(t[h][m], t[h][m], att[h]);
                                    ats[h] = __fmaf_rn(t[h][m], q[h][m], ats[h]);
                                }
                            }
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        if (!U.on[h]) continue;
                        float tt, ts;
                        lanes_tree_sum2<float>(att[h], ats[h], lane, reinterpret_cast<float *>(sm[gi]), tt, ts, gsync);
                        if (lane == 0) reinterpret_cast<double2 *>(U.S(A, h).part)[U.lc[h]] = make_double2(tt, ts);
                    }
                }
            });
            if (!grid_sync(bar, target, &s_ok)) break;
            two_sums(0);
            if (threadIdx.x < A.nsys && inner_active(sst[threadIdx.x], sdc[threadIdx.x])) {
                const double ftt = s_sum[threadIdx.x][0];
                sst[threadIdx.x].w = (ftt > 0.0) ? s_sum[threadIdx.x][1] / ftt : 0.0;
            }
            __syncthreads();
            // r = s - w t; <r0, r>, <r, r>
            unit_phase([&](auto units) {
                constexpr int H = decltype(units)::value;
                for (int u = cbegin; u < total_units; u += H * gstride) {
                    const UnitPair<CAP, H> U(A, sst, sdc, u, gstride, total_units);
                    if (U.none()) continue;
                    float t[H][MRPL], sv[H][MRPL], q[H][MRPL];
#pragma unroll
                    for (int h = 0; h < H; ++h)
#pragma unroll
                        for (int m = 0; m < MRPL; ++m) {
                            const int row = U.lc[h] * MUNIT + lane + m * LANES;
                            t[h][m] = U.S(A, h).t[row];
                            sv[h][m] = U.S(A, h).s[row];
                            q[h][m] = U.S(A, h).r0[row];
                        }
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        if (!U.on[h]) continue;
                        const float w = (float)sst[U.si[h]].w;
                        float a0r = 0.0f, arr = 0.0f;
#pragma unroll
                        for (int m = 0; m < MRPL; ++m) {
                            const int row = U.lc[h] * MUNIT + lane + m * LANES;
                            const float r = __fmaf_rn(-w, t[h][m], sv[h][m]);
                            U.S(A, h).r[row] = r;
                            if (row < U.S(A, h).n) {
                                a0r = __fmaf_rn(q[h][m], r, a0r);
                                arr = __fmaf_rn(r, r, arr);
                            }
                        }
                        float t0r, trr;
                        lanes_tree_sum2<float>(a0r, arr, lane, reinterpret_cast<float *>(sm[gi]), t0r, trr, gsync);
                        if (lane == 0)
                            reinterpret_cast<double2 *>(U.S(A, h).part + 2 * (size_t)U.S(A, h).nchunks * MSUB)[U.lc[h]] =
                                make_double2(t0r, trr);
                    }
                }
            });
            grid_arrive(bar, target);
            // x += alpha y + w z, while the other blocks arrive.  The loop may end
            // behind this barrier, which does not order what is written here: in
            // this launch an element of x is read by the thread that wrote it, and
            // by no other (each_chunk).
            stream_chunks([&](int si, const MSys &S, int i) {
                const float alpha = (float)sst[si].alpha, w = (float)sst[si].w;
                const float4 x = at4(S.x, i), y = at4(S.y, i), z = at4(S.z, i);
                const float4 xn = each4(
                    [&](float x1, float y1, float z1) { return __fmaf_rn(w, z1, __fmaf_rn(alpha, y1, x1)); }, x, y, z);
                return Pair4{S.x, nullptr, xn, xn};
            });
            if (!grid_wait(bar, target, &s_ok)) break;
            two_sums(2);
            if (threadIdx.x < A.nsys && inner_active(sst[threadIdx.x], sdc[threadIdx.x]))
                m32_end_iteration(sst[threadIdx.x], s_sum[threadIdx.x][0], s_sum[threadIdx.x][1]);
            __syncthreads();
        }
        bool any = false;
        if constexpr (CAP <= KMAX) {
            for (int q = 0; q < A.nsys; ++q) any = any || inner_active(sst[q], sdc[q]);
        } else {  // the lanes of each warp split the systems
            for (int q = threadIdx.x & 31; q < A.nsys; q += 32) any = any || inner_active(sst[q], sdc[q]);
            any = __any_sync(0xffffffffu, any);
        }
        if (!any) {
            ++it;
            break;
        }
    }
    // the correction in FP64, for k_dc_step and k_dc_update: one conversion and
    // product per row here instead of one per operand there
    __shared__ double s_inv[CAP];
    if (threadIdx.x < A.nsys) s_inv[threadIdx.x] = 1.0 / A.sys[threadIdx.x].dc->scale;
    __syncthreads();
    // (each element by the thread that last updated x there)
    auto corrected = [&](int si) { return !sdc[si] && sst[si].info == 0; };
    if constexpr (FUSED) {
        for (int u = cbegin; u < total_units; u += gstride) {
            const int si = msys_of_chunk(A, u / MSUB);
            if (!corrected(si)) continue;
            const MSys &S = A.sys[si];
            const int r0 = (u - S.chunk_begin * MSUB) * MUNIT + lane;
            float x[MRPL];
#pragma unroll
            for (int m = 0; m < MRPL; ++m) x[m] = S.x[r0 + m * LANES];
#pragma unroll
            for (int m = 0; m < MRPL; ++m) S.d64[r0 + m * LANES] = (double)x[m] * s_inv[si];
        }
    } else {
        each_chunk(corrected, [&](int si, const MSys &S, int i) {
            const float4 x[2] = {at4(S.x, i), at4(S.x, i + LANES)};
            const double inv = s_inv[si];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double2 *const d = reinterpret_cast<double2 *>(S.d64) + 2 * (i + h * LANES);
                d[0] = make_double2((double)x[h].x * inv, (double)x[h].y * inv);
                d[1] = make_double2((double)x[h].z * inv, (double)x[h].w * inv);
            }
        });
    }
    if (blockIdx.x == 0 && threadIdx.x < A.nsys) {
        KState k = sst[threadIdx.x];
        k.counter = 0;
        *A.sys[threadIdx.x].st = k;
    }
}

// Step length of the round's correction delta = double(d) / scale (S.d64):
// theta = <r64, A64 delta> / <A64 delta, A64 delta> minimizes the FP64
// residual along delta, so a correction from an inaccurate FP32 solve can
// shrink the residual less but never grow it.  The last block to finish
// sets dc->theta.
template <int CAP, int G>
__global__ void __launch_bounds__(LANES *G, 8 / G) k_dc_step(const __grid_constant__ MSetArgT<CAP> A) {
    __shared__ double s_q[CH], s_r[CH], sm[8];
    __shared__ int sh[4];
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {
        const MSys &S = A.sys[msys_of_chunk(A, c)];
        if (!(__ldcg(&S.dc->done) == 0 && __ldcg(&S.st->info) == 0)) continue;
        const int lc = c - S.chunk_begin;
#pragma unroll
        for (int i = 0; i < RPL / G; ++i) {
            const int q = lane + (gi * (RPL / G) + i) * LANES, row = lc * CH + q;
            s_q[q] = spmv_f64_row(S, row, S.d64);
            s_r[q] = S.r64[row];
        }
        __syncthreads();
        for (int j = gi; j < 2; j += G) {
            const double t = lanes_tree_sum<double>(lane_dot(j == 0 ? s_r : s_q, s_q, lane, min(CH, S.n - lc * CH)), lane,
                                                    sm + 4 * j, GroupSync{gi + 1});
            if (lane == 0) S.part[2 * (size_t)lc + j] = t;
        }
        if (m_arrive_last(&S.dc->counter, (unsigned)S.nchunks, sh) && threadIdx.x < LANES) {
            double frq, fqq;
            lanes_final_sum2(S.part, S.nchunks, lane, sm, frq, fqq, GroupSync{1});
            if (threadIdx.x == 0) {
                S.dc->counter = 0;
                const double th = (fqq > 0.0) ? frq / fqq : 0.0;
                S.dc->theta = finite(th) ? th : 0.0;
            }
        }
    }
}

template <int CAP>
__global__ void k_dc_update(const __grid_constant__ MSetArgT<CAP> A) {
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {
        const MSys &S = A.sys[msys_of_chunk(A, c)];
        if (!(__ldcg(&S.dc->done) == 0 && __ldcg(&S.st->info) == 0)) continue;
        const double theta = __ldcg(&S.dc->theta);
        const int r0 = (c - S.chunk_begin) * CH + threadIdx.x;
        double d[RPL], x[RPL];
#pragma unroll
        for (int m = 0; m < RPL; ++m) {  // all loads before the first store
            d[m] = S.d64[r0 + m * LANES];
            x[m] = S.x64[r0 + m * LANES];
        }
#pragma unroll
        for (int m = 0; m < RPL; ++m) S.x64[r0 + m * LANES] = __fma_rn(theta, d[m], x[m]);
    }
}

#undef NS3D_MCHUNK_LOOP

void launch_mg_galerkin(const MSys &S, cudaStream_t st) {
    for (int k = 1; k <= S.mg.nlev; ++k) {
        const MGLevel &C = S.mg.lev[k];
        const int npad_f = k == 1 ? S.npad : S.mg.lev[k - 1].npad;
        const int *nbr_f = k == 1 ? S.nbr : S.mg.lev[k - 1].nbr;
        const float *coef_f = k == 1 ? S.coef32 : S.mg.lev[k - 1].coef;
        count_launches(1);
        k_mg_galerkin<<<std::max(1, std::min((C.n + 31) / 32, 152 * 8)), 256, 0, st>>>(npad_f, nbr_f, coef_f, C);
    }
}

// FP32 copy of a system's coefficients and inverse diagonal (npad is a
// multiple of 1024 and both arrays come from the pool, so pairs are aligned)
__global__ void k_to_f32(const double2 *__restrict__ coef, const double2 *__restrict__ invdiag, int pairs,
                         float2 *__restrict__ coef32, float2 *__restrict__ invdiag32) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += gridDim.x * blockDim.x) {
        double2 v[8];
#pragma unroll
        for (int s = 0; s < 7; ++s) v[s] = coef[(size_t)s * pairs + i];
        v[7] = invdiag[i];
#pragma unroll
        for (int s = 0; s < 7; ++s) coef32[(size_t)s * pairs + i] = make_float2((float)v[s].x, (float)v[s].y);
        invdiag32[i] = make_float2((float)v[7].x, (float)v[7].y);
    }
}

// ---- launchers ------------------------------------------------------------------
static inline int m_grid(int total_chunks) { return std::max(1, std::min(total_chunks, device_sm_count() * 32)); }

void launch_to_f32(const double *coef, const double *invdiag, int npad, float *coef32, float *invdiag32,
                   cudaStream_t st) {
    const int pairs = npad / 2;
    count_launches(1);
    k_to_f32<<<std::min((pairs + 255) / 256, device_sm_count() * 32), 256, 0, st>>>(
        reinterpret_cast<const double2 *>(coef), reinterpret_cast<const double2 *>(invdiag), pairs,
        reinterpret_cast<float2 *>(coef32), reinterpret_cast<float2 *>(invdiag32));
}

template <int CAP>
void launch_dc_resid(const MSetArgT<CAP> &A, int first, cudaStream_t st) {
    if (A.total_chunks <= 0) return;
    count_launches(1);
    if (wide_chunks(A.total_chunks, device_sm_count()))
        k_dc_resid<CAP, WIDE_G><<<m_grid(A.total_chunks), LANES * WIDE_G, 0, st>>>(A, first);
    else
        k_dc_resid<CAP, NARROW_G><<<m_grid(A.total_chunks), LANES * NARROW_G, 0, st>>>(A, first);
    if (first) {
        count_launches(1);
        k_dc_zero<CAP><<<m_grid(A.total_chunks), LANES, 0, st>>>(A);
    }
}

template <int CAP>
void launch_m32_init(const MSetArgT<CAP> &A, cudaStream_t st) {
    if (A.total_chunks <= 0) return;
    count_launches(1);
    if (wide_chunks(A.total_chunks, device_sm_count()))
        k_m32_init<CAP, WIDE_G><<<m_grid(A.total_chunks), LANES * WIDE_G, 0, st>>>(A);
    else
        k_m32_init<CAP, 1><<<m_grid(A.total_chunks), LANES, 0, st>>>(A);  // bytes only: 74 us at 10.5 M rows, 101 with two groups
}


// Sets up to kFusedRows rows run the three-phase loop (fewer barriers; the
// recomputed neighbour operands are cache hits), larger ones the five-phase
// loop (157 K rows: 47 ms three-phase, 51 five-phase for two SIMPLER outer
// iterations; 498 K rows: 100 and 88 ms for one SIMPLERR outer iteration).
constexpr long kFusedRows = 1L << 18;

// (the V-cycle runs in the five-phase loop)
bool m32_fused(long rows, bool mg) { return rows <= kFusedRows && !mg; }

// at most 21 words a row and one more a level (mg_tail_words)
constexpr size_t kTailSmemMax = ((size_t)21 * MG_TAIL_ROWS + MG_MAX) * 4;

// Sets without a multilevel system whose share of the SMs gives every chunk a
// block run the loop with resident chunks (mixed_chunk.cuh).  Ten SIMPLEC
// outer iterations of a 56^3 image (pressure 103 chunks): 85 -> 68 ms.
template <int CAP>
void plan_mixed(MSetArgT<CAP> &A, int share) {
    A.resident = 0;
    for (int i = 0; i < A.nsys; ++i)
        if (A.sys[i].mg.nlev > 0) return;
    const int sharers = CAP > KMAX ? std::max(share, 1) : std::max(1, active_solves());
    A.resident = A.total_chunks <= std::max(1, device_sm_count() / sharers);
}

template <int CAP>
static cudaError_t launch_m32_resident(const MSetArgT<CAP> &A, GridBar *bar, int max_iters, cudaStream_t st) {
    const void *fn = (const void *)k_m32_chunk<CAP>;
    static std::atomic<bool> ready{false};
    cudaError_t e = cudaSuccess;
    if (!ready.load()) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMChunkSmemBytes);
        if (e != cudaSuccess) return e;
        ready = true;
    }
    e = reset_grid_bar(bar, st);
    if (e != cudaSuccess) return e;
    MSetArgT<CAP> a = A;
    void *args[] = {&a, &bar, &max_iters};
    count_launches(1);
    return cudaLaunchCooperativeKernel(fn, A.total_chunks, CH, args, kMChunkSmemBytes, st);
}

template <int CAP>
cudaError_t launch_m32_loop(const MSetArgT<CAP> &A, GridBar *bar, int max_iters, cudaStream_t st, int variant,
                            int share) {
    if (A.total_chunks <= 0 || max_iters <= 0) return cudaSuccess;
    if (A.resident) return launch_m32_resident(A, bar, max_iters, st);
    long rows = 0;
    bool mg = false;
    for (int i = 0; i < A.nsys; ++i) {
        rows += A.sys[i].n;
        mg = mg || A.sys[i].mg.nlev > 0;
    }
    const bool fused = variant < 0 ? m32_fused(rows, mg) : (variant == 1 && !mg);
    const bool packed = CAP <= KMAX && A.sys[0].mg.nlev > 0 && A.sys[0].mg.pack;
    const void *fn = fused ? (const void *)k_m32_loop<true, CAP> : (const void *)k_m32_loop<false, CAP>;
    if constexpr (CAP <= KMAX)
        if (packed) fn = (const void *)k_m32_loop<false, CAP, true>;
    static std::atomic<int> occ_cache[3];
    const int form = packed ? 2 : fused;
    const size_t tail_max = CAP <= KMAX && !fused ? kTailSmemMax : 0;
    const size_t smem = tail_max && A.sys[0].mg.nlev > 0 ? mg_tail_words(A.sys[0].mg) * 4 : 0;
    int occ = occ_cache[form].load();
    if (occ == 0) {
        cudaError_t e = cudaSuccess;
        if (tail_max) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tail_max);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, LOOP_THREADS, tail_max);
        if (e != cudaSuccess) return e;
        if (occ <= 0) return cudaErrorLaunchOutOfResources;
        occ_cache[form] = occ;
    }
    // a merged set (many solves' systems) spreads over its share of the SMs
    const int grid = CAP > KMAX
                         ? std::max(1, std::min(A.total_chunks * MSUB, device_sm_count() * occ / std::max(share, 1)))
                         : loop_grid(A.total_chunks * MSUB, MSUB, occ);
    cudaError_t e = reset_grid_bar(bar, st);
    if (e != cudaSuccess) return e;
    MSetArgT<CAP> a = A;
    void *args[] = {&a, &bar, &max_iters};
    count_launches(1);
    return cudaLaunchCooperativeKernel(fn, grid, LOOP_THREADS, args, smem, st);
}

template <int CAP>
void launch_dc_update(const MSetArgT<CAP> &A, cudaStream_t st) {
    if (A.total_chunks <= 0) return;
    count_launches(2);
    if (wide_chunks(A.total_chunks, device_sm_count()))
        k_dc_step<CAP, WIDE_G><<<m_grid(A.total_chunks), LANES * WIDE_G, 0, st>>>(A);
    else
        k_dc_step<CAP, NARROW_G><<<m_grid(A.total_chunks), LANES * NARROW_G, 0, st>>>(A);
    k_dc_update<CAP><<<m_grid(A.total_chunks), LANES, 0, st>>>(A);
}

template void plan_mixed<KMAX>(MSetArg &, int);
template void plan_mixed<KMAX_MERGED_M>(MSetArgMerged &, int);
template void launch_dc_resid<KMAX>(const MSetArg &, int, cudaStream_t);
template void launch_dc_resid<KMAX_MERGED_M>(const MSetArgMerged &, int, cudaStream_t);
template void launch_m32_init<KMAX>(const MSetArg &, cudaStream_t);
template void launch_m32_init<KMAX_MERGED_M>(const MSetArgMerged &, cudaStream_t);
template cudaError_t launch_m32_loop<KMAX>(const MSetArg &, GridBar *, int, cudaStream_t, int, int);
template cudaError_t launch_m32_loop<KMAX_MERGED_M>(const MSetArgMerged &, GridBar *, int, cudaStream_t, int, int);
template void launch_dc_update<KMAX>(const MSetArg &, cudaStream_t);
template void launch_dc_update<KMAX_MERGED_M>(const MSetArgMerged &, cudaStream_t);

}  // namespace ns3d
