// krylov.cu -- batched Jacobi-preconditioned BiCGSTAB on the device.
//
// Replaces Eigen::BiCGSTAB<SparseMatrix<double,RowMajor>> with the default
// DiagonalPreconditioner (src/NSBase.h:97-100), called through
// solveWithGuess at src/NSBase.cxx:1799,1825,1852,2343,2393,2397.  The
// algorithm is the published right-preconditioned BiCGSTAB
// (van der Vorst 1992) with the behaviour the reference depends on:
// convergence when |r|^2 <= tol^2 |b|^2, iterations() counting completed
// iterations, error() = |r|/|b|, restart with a fresh shadow residual when
// |rho| < eps^2 |r0|^2 (the counter restarts on the first restart), and the
// zero right-hand side rule (x = 0, Success, iterations() = max).
//
// A solve set holds up to KMAX independent systems (the three momentum
// components, or the pressure system).  Their rows are processed as one list
// of 1024-row chunks; the set is passed to every kernel by value
// (__grid_constant__), so a block finds its system and the system's arrays
// in constant memory.  One BiCGSTAB iteration has five phases:
//   K1 p = r + beta (p - w v); y = D^-1 p
//   K2 v = A y, <r0,v>                      -> alpha
//   K3 s = r - alpha v; z = D^-1 s
//   K4 t = A z, <t,t>, <t,s>                -> w
//   K5 x += alpha y + w z; r = s - w t, <r0,r>, <r,r> -> convergence, beta
// All iterations of a solve run in one persistent cooperative launch:
// k_kr_loop, the phases separated by bounded grid barriers (loop.cuh), or for
// sets of at most one chunk per SM k_kr_chunk (krylov_chunk.cuh, included
// below), which needs none.
// The set-up (r = b - A x, norms) and the restart after |rho| breakdown are
// separate launches whose last block to finish (one atomic counter per
// system) combines the partials, so they wait on no other block.
#include <atomic>
#include <cfloat>
#include <cstring>

#include "device.cuh"
#include "kernels.h"
#include "loop.cuh"

namespace ns3d {

// ---- tensor memory as a resident store --------------------------------------
// The 256 KB of tensor memory of an SM lie idle in this solver.  The loop
// kernel keeps matrix coefficients there for a launch: a warp reaches the 32
// lanes of its rank in the warpgroup, a group of 128 threads has 64 of the 512
// columns, so a thread owns 64 words, and reads back what it wrote itself.
// A row's first NT coefficients take 2 NT words, padded to TMEM_ROW<NT>.
// With four of seven coefficients there a row's data outside the SM shrink
// from 136 to 104 bytes, and 1.05 M rows fit the L2: 79.5 -> 72.8 us per
// iteration (0.73 M rows 58.1 -> 55.8).  With several chunks per group only
// the first could live there: 3.55 M rows 250 -> 253 us, so not used.
constexpr int TMEM_COLUMNS = 512;
template <int NT>
constexpr int TMEM_ROW = NT > 4 ? 16 : 8;

// one warp of the block; *base (shared) receives the address
__device__ __forceinline__ void tmem_alloc(unsigned int *base) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (unsigned int)__cvta_generic_to_shared(base)),
                 "n"(TMEM_COLUMNS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
// the same warp, after every other warp's last access
__device__ __forceinline__ void tmem_free(unsigned int base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(TMEM_COLUMNS) : "memory");
}
// NT doubles to / from the words at taddr (whole warps)
template <int NT>
__device__ __forceinline__ void tmem_store(unsigned int taddr, const double *c) {
    unsigned int w[16];
    __syncwarp();  // .aligned: the whole warp issues the instruction
#pragma unroll
    for (int d = 0; d < 8; ++d) {
        w[2 * d] = d < NT ? (unsigned int)__double2loint(c[d < NT ? d : 0]) : 0u;
        w[2 * d + 1] = d < NT ? (unsigned int)__double2hiint(c[d < NT ? d : 0]) : 0u;
    }
    if constexpr (NT > 4)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15, %16};" ::"r"(taddr),
            "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]),
            "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
            : "memory");
    else if constexpr (NT > 0)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                     "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
}
template <int NT>
__device__ __forceinline__ void tmem_load(unsigned int taddr, double *c) {
    unsigned int w[16];
    if (NT > 0) __syncwarp();
    if constexpr (NT > 4)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
            "%15}, [%16];\n tcgen05.wait::ld.sync.aligned;"
            : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]),
              "=r"(w[8]), "=r"(w[9]), "=r"(w[10]), "=r"(w[11]), "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15])
            : "r"(taddr)
            : "memory");
    else if constexpr (NT > 0)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
            " tcgen05.wait::ld.sync.aligned;"
            : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
            : "r"(taddr)
            : "memory");
#pragma unroll
    for (int d = 0; d < NT; ++d) c[d] = __hiloint2double((int)w[2 * d + 1], (int)w[2 * d]);
}

struct Row4 {  // a thread's RPL rows
    double v[RPL];
};

// A thread's rows are r0 + m*LANES, m < RPL (coalesced across the warp).
__device__ __forceinline__ Row4 ld4(const double *p) {
    Row4 r;
#pragma unroll
    for (int m = 0; m < RPL; ++m) r.v[m] = p[m * LANES];
    return r;
}
__device__ __forceinline__ void st4(double *p, const Row4 &r) {
#pragma unroll
    for (int m = 0; m < RPL; ++m) p[m * LANES] = r.v[m];
}

// One row of y = A x: fma chain in ascending column order from 0 (the order
// of row_ordered in device.cuh).  Every gather is issued unconditionally (a
// missing neighbour reads the row's own element) so the loads of a row do
// not wait on each other; only the fused multiply-adds are predicated.  The
// two rare orders (W directly before the row, E directly after it) are taken
// only by warps that contain such a row.
// The neighbour columns come from `nb` (nb[k * stride], k = slot - 1): the
// system's table in global memory, or a chunk's copy in shared memory.  The
// first NT coefficients (slots P, W, E, ...) come from the tensor memory of
// the SM (taddr; tmem_row below), the others from memory.
template <int NT, class Stride>
__device__ __forceinline__ double spmv_row_nb(const KSys &S, int row, const double *__restrict__ x, const int *nb,
                                              Stride stride, unsigned int taddr = 0) {
    const size_t np = (size_t)S.npad;
    const double *cf = S.coef + row;
    const int nW = nb[0 * stride], nE = nb[1 * stride], nS = nb[2 * stride], nN = nb[3 * stride],
              nB = nb[4 * stride], nT = nb[5 * stride];
    const double xP = x[row];
    const double xW = x[nW >= 0 ? nW : row], xE = x[nE >= 0 ? nE : row], xS = x[nS >= 0 ? nS : row];
    const double xN = x[nN >= 0 ? nN : row], xB = x[nB >= 0 ? nB : row], xT = x[nT >= 0 ? nT : row];
    double cc[7];
#pragma unroll
    for (int d = NT; d < 7; ++d) cc[d] = ro(cf + d * np);
    tmem_load<NT>(taddr, cc);
    const double cP = cc[0], cW = cc[1], cE = cc[2], cS = cc[3], cN = cc[4], cB = cc[5], cT = cc[6];
    const bool wlate = nW >= 0 && nW == row - 1;
    const bool eearly = nE >= 0 && nE == row + 1;
    double acc = 0.0;
    if (__any_sync(0xffffffffu, wlate || eearly)) {
        if (!wlate && nW >= 0) acc = __fma_rn(cW, xW, acc);
        if (nS >= 0) acc = __fma_rn(cS, xS, acc);
        if (nB >= 0) acc = __fma_rn(cB, xB, acc);
        if (wlate) acc = __fma_rn(cW, xW, acc);
        acc = __fma_rn(cP, xP, acc);
        if (eearly) acc = __fma_rn(cE, xE, acc);
        if (nT >= 0) acc = __fma_rn(cT, xT, acc);
        if (nN >= 0) acc = __fma_rn(cN, xN, acc);
        if (!eearly && nE >= 0) acc = __fma_rn(cE, xE, acc);
    } else {
        if (nW >= 0) acc = __fma_rn(cW, xW, acc);
        if (nS >= 0) acc = __fma_rn(cS, xS, acc);
        if (nB >= 0) acc = __fma_rn(cB, xB, acc);
        acc = __fma_rn(cP, xP, acc);
        if (nT >= 0) acc = __fma_rn(cT, xT, acc);
        if (nN >= 0) acc = __fma_rn(cN, xN, acc);
        if (nE >= 0) acc = __fma_rn(cE, xE, acc);
    }
    return acc;
}

__device__ __forceinline__ double spmv_row(const KSys &S, int row, const double *__restrict__ x) {
    return spmv_row_nb<0>(S, row, x, S.nbr + row, (size_t)S.npad);
}

// the same from a chunk's 16-bit distances (nb16[k * CH]: |column - row| of
// slot k + 1, 0 = no entry): W, S and B columns lie before the row, E, N and
// T columns after it
template <int NT>
__device__ __forceinline__ double spmv_row_16(const KSys &S, int row, const double *__restrict__ x,
                                              const unsigned short *nb16, unsigned int taddr) {
    int nb[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int d = nb16[k * CH];
        nb[k] = d == 0 ? -1 : row + ((k & 1) ? d : -d);
    }
    return spmv_row_nb<NT>(S, row, x, nb, 1, taddr);
}

// y = A x for the thread's rows (rows >= n give garbage that callers mask)
__device__ __forceinline__ Row4 spmv4(const KSys &S, int r0, const double *__restrict__ x) {
    Row4 out;
#pragma unroll
    for (int m = 0; m < RPL; ++m) out.v[m] = spmv_row(S, r0 + m * LANES, x);
    return out;
}

// system owning global chunk c (chunk_begin ascending, first system begins
// at 0; a system without rows shares its chunk_begin with the next one, and
// both forms pick the last system whose first chunk is <= c)
template <int CAP>
__device__ __forceinline__ int sys_of_chunk(const KSetArgT<CAP> &A, int c) {
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

// the done/paused flags change only between kernels (or after the last
// chunk of the system arrived), so every thread of a block reads the same
__device__ __forceinline__ bool sys_active(const KSys &S) {
    return (__ldcg(&S.st->done) | __ldcg(&S.st->paused)) == 0;
}

__device__ __forceinline__ bool arrive_last(KState *st, unsigned int total, int *sh) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int prev = atomicAdd(&st->counter, 1u);
        sh[0] = (prev == total - 1) ? 1 : 0;
    }
    __syncthreads();
    bool last = sh[0] != 0;
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ void finish_loop(KState *st) {
    // loop exit: error() and info() as Eigen reports them
    st->done = 1;
    st->error = sqrt(st->rr / st->rhs_sqnorm);
    st->info = (st->error <= st->tol) ? 0 : 2;
}

__device__ __forceinline__ bool state_active(const KState &k) { return (k.done | k.paused) == 0; }

}  // namespace ns3d
#include "krylov_chunk.cuh"
namespace ns3d {

#define NS3D_CHUNK_LOOP                                                        \
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {            \
        const int sidx = sys_of_chunk(A, c);                                   \
        const KSys &S = A.sys[sidx];                                           \
        const int lc = c - S.chunk_begin;                                      \
        const int r0 = lc * CH + threadIdx.x;

// r = b - A x into S.r and S.r0 for a chunk's rows, |r|^2 and (BB) |b|^2 of the
// chunk into its partials.  sm: 2 CH operands, 8 for the trees (also of the
// final sum, during which the other groups may already write the next chunk's
// operands).
template <int G, bool BB>
__device__ __forceinline__ void chunk_residual(const KSys &S, int lc, double *sm) {
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    double *const s_r = sm, *const s_b = sm + CH;
#pragma unroll
    for (int i = 0; i < RPL / G; ++i) {
        const int q = lane + (gi * (RPL / G) + i) * LANES, row = lc * CH + q;
        const double b = S.b[row];
        const double r = b - spmv_row(S, row, S.x);
        s_r[q] = r;
        if (BB) s_b[q] = b;
        S.r[row] = r;
        S.r0[row] = r;
    }
    __syncthreads();
    // sum j by group j (by group 0 in turn when it is the only one)
    for (int j = gi; j < (BB ? 2 : 1); j += G) {
        const double *v = j == 0 ? s_r : s_b;
        const double t = lanes_tree_sum<double>(lane_dot(v, v, lane, min(CH, S.n - lc * CH)), lane, sm + 2 * CH + 4 * j,
                                                GroupSync{gi + 1});
        if (lane == 0) S.part[2 * (size_t)lc + j] = t;
    }
}

// ---- init: r = b - A x, r0 = r, |r|^2, |b|^2 ---------------------------------
template <int CAP, int G>
__global__ void __launch_bounds__(LANES *G, 8 / G) k_kr_init(const __grid_constant__ KSetArgT<CAP> A) {
    __shared__ double sm[2 * CH + 8];
    __shared__ int sh[2];
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {
        const KSys &S = A.sys[sys_of_chunk(A, c)];
        const int lc = c - S.chunk_begin;
        chunk_residual<G, true>(S, lc, sm);
        if (arrive_last(S.st, (unsigned)S.nchunks, sh) && threadIdx.x < LANES) {
            double rr, bb;
            lanes_final_sum2(S.part, S.nchunks, threadIdx.x, sm + 2 * CH, rr, bb, GroupSync{1});
            if (threadIdx.x == 0) {
                KState *st = S.st;
                st->counter = 0;
                st->r0_sqnorm = rr;
                st->rr = rr;
                st->rhs_sqnorm = bb;
                st->iter = 0;
                st->restarts = 0;
                st->paused = 0;
                st->zero_rhs = 0;
                if (bb == 0.0) {
                    st->zero_rhs = 1;
                    st->done = 1;
                    st->iter = st->maxit;
                    st->error = st->tol;
                    st->info = 0;
                } else {
                    st->rho = 1.0;
                    st->alpha = 1.0;
                    st->w = 1.0;
                    st->tol2 = st->tol * st->tol * bb;
                    if (!(rr > st->tol2 && 0 < st->maxit)) {
                        finish_loop(st);
                    } else {
                        // first iteration: rho = <r0, r> equals |r0|^2 bit for bit
                        const double rho_old = st->rho;
                        const double rho = rr;
                        st->beta = (rho / rho_old) * (st->alpha / st->w);
                        st->rho = rho;
                        st->done = 0;
                    }
                }
            }
        }
    }
}

// p = v = 0; x = 0 for a zero right-hand side; what the one-chunk-per-block
// loop exchanges (krylov_chunk.cuh)
template <int CAP>
__global__ void k_kr_init2(const __grid_constant__ KSetArgT<CAP> A) {
    NS3D_CHUNK_LOOP
        Row4 z;
#pragma unroll
        for (int m = 0; m < RPL; ++m) z.v[m] = 0.0;
        st4(S.p + r0, z);
        st4(S.v + r0, z);
        if (A.one_per_block) {
            for (double *q : {S.y, S.s, S.z, S.t}) st4(q + r0, z);
            if (threadIdx.x < TAG_KINDS) {
                unsigned long long *slot = chunk_tag_words(S) + 2 * ((size_t)threadIdx.x * S.nchunks + lc);
                slot[0] = slot[1] = 0;
                if (lc == 0) *tag_counter(S.part, S.nchunks, threadIdx.x) = 0;
            }
        }
        if (__ldcg(&S.st->zero_rhs)) st4(S.x + r0, z);
    }
}

// ---- the BiCGSTAB iteration loop: one persistent cooperative kernel ----------
//
// LOOP_THREADS threads per block form LOOP_GROUPS groups of LANES threads; a
// chunk is worked on by GPC groups (the lanes own the rows of the fixed
// reduction order) and reduced with a named barrier.  Every block keeps a copy
// of the per-system scalars in shared memory; after each grid-wide barrier
// every block combines the chunk partials of each system in the fixed order
// itself (group g for systems g, g + LOOP_GROUPS, ...), so all copies stay
// bit-identical without a broadcast.  Partials of the three reductions of an
// iteration go to separate regions of S.part, so a block that runs ahead never
// overwrites partials another block is still combining:
//   [0, 2n)  <t,t>, <t,s> pairs     [2n, 4n)  <r0,r>, <r,r> pairs
//   [4n, 5n) <r0,v>
// The loop ends when every system is done, when a system needs a restart
// (the host recomputes its residual and launches the loop again), after
// `max_iters` iterations, or when a grid barrier gives up waiting.
//
// GPC 0: any number of chunks per group (group g of the grid takes chunks
// g, g + groups, ...).  GPC 1, 2, 4: one chunk per GPC groups and no more, so
// a set of 1.2 to 4 chunks per SM does not leave half of the groups idle: a
// chunk's rows are split over its groups (group p takes the lanes' rows
// p RPL / GPC ...), and the lanes' sums pass from group to group through
// shared memory, in row order (eight images in lockstep, pressure sets of
// about 480 chunks: 185 -> 168 ms).
//
// Loads come in batches before the first store of the batch: the vectors may
// alias for the compiler, so a store between them would make every row wait
// for its own loads (K1, K3 and K5 took 12.5, 11.5 and 17.0 us at 1.05 M rows
// that way, 9.8, 7.0 and 16.1 in batches).  x is updated between the two
// halves of the last barrier, in time the block would spend waiting.
constexpr int kSpmvUnroll = 2;  // rows in flight per thread in the SpMV phases (1: 1% slower, 4: 3%)

// Resident neighbour tables (GPC > 0).  The matrix does not change during a
// solve, so the block keeps its chunks' columns in shared memory as 16-bit
// distances from the row (12 KB a chunk): 48 B less traffic per row-iteration
// and no index load before the gathers.  Columns further than 65535 rows away
// are read from memory, a group's rows at a time.  With GPC 0 the tables of
// one chunk would only take L1 from all: 32-bit tables of the first chunk
// (192 KB) made an iteration of 3.55 M rows 291 us instead of 252.
template <int GPC>
constexpr size_t kNbrSmemBytes = GPC ? (size_t)(LOOP_GROUPS / (GPC ? GPC : 1)) * 6 * CH * sizeof(unsigned short) : 0;

template <int CAP, int GPC>
__global__ void __launch_bounds__(LOOP_THREADS, LOOP_MIN_BLOCKS)
    k_kr_loop(const __grid_constant__ KSetArgT<CAP> A, GridBar *bar, LoopProf *prof, int max_iters) {
    static_assert(CAP <= LOOP_THREADS, "one thread copies each system's state");
    constexpr bool RES = GPC > 0;
    constexpr int PARTS = RES ? GPC : 1, RP = RPL / PARTS, BATCH = RP < 4 ? RP : 4;
    // a row's coefficients in tensor memory: a thread's 64 words hold RP rows
    constexpr int NT = RES ? (RP < 8 ? 7 : 4) : 0;
    static_assert(!RES || RP * TMEM_ROW<NT> <= TMEM_COLUMNS / LOOP_GROUPS, "a thread's words");
    __shared__ KState sst[CAP];
    __shared__ double sm[LOOP_GROUPS][16];
    __shared__ double s_acc[PARTS > 1 ? LOOP_GROUPS : 1][2][LANES];  // the lanes' sums on their way
    __shared__ int s_ok;
    __shared__ unsigned int s_tmem;
    extern __shared__ unsigned short s_nbr_all[];  // RES: [LOOP_GROUPS / GPC][6][CH]
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES, part = gi % PARTS;
    const GroupSync gsync{gi + 1};
    // chunk c belongs to block c % gridDim.x: every block, hence every SM,
    // gets the same number of chunks to within one
    const int gstride = gridDim.x * LOOP_GROUPS;
    const int cbegin = blockIdx.x + gridDim.x * (gi / PARTS);
    const int lane0 = part * RP * LANES + lane;  // the thread's first row in a chunk
    if (threadIdx.x < A.nsys) sst[threadIdx.x] = *A.sys[threadIdx.x].st;
    bool far = false;  // RES: a row of the group has a column beyond 16 bits
    unsigned short *const s_nbr = s_nbr_all + (size_t)(gi / PARTS) * 6 * CH + lane0;
    if (RES && cbegin < A.total_chunks) {  // the group's rows, for the whole launch
        const KSys &S = A.sys[sys_of_chunk(A, cbegin)];
        const int row0 = (cbegin - S.chunk_begin) * CH + lane0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
#pragma unroll
            for (int m = 0; m < RP; ++m) {
                const int row = row0 + m * LANES, c = ro(S.nbr + (size_t)k * S.npad + row);
                const int d = c < 0 ? 0 : (k & 1) ? c - row : row - c;
                far = far || d < 0 || d > 65535;
                s_nbr[k * CH + m * LANES] = (unsigned short)d;
            }
        int any;  // over the group's 128 threads
        asm volatile(
            "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n barrier.cta.red.or.pred q, %2, %3, p;\n"
            " selp.s32 %0, 1, 0, q;\n}"
            : "=r"(any)
            : "r"((int)far), "r"(gi + 1), "n"(LANES)
            : "memory");
        far = any != 0;
    }
    unsigned int target = grid_sync_start(bar);  // the counter is zeroed before every launch
    if (RES && threadIdx.x < 32) tmem_alloc(&s_tmem);
    if (RES) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the scalar copies in sst are complete, the tensor memory is allocated
    if (RES) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // the words of the thread's rows
    const unsigned int taddr = RES ? s_tmem + ((unsigned int)(lane & ~31) << 16) + gi * (TMEM_COLUMNS / LOOP_GROUPS) : 0;
    if (RES && cbegin < A.total_chunks) {
        const KSys &S = A.sys[sys_of_chunk(A, cbegin)];
        const int row0 = (cbegin - S.chunk_begin) * CH + lane0;
#pragma unroll 1
        for (int m = 0; m < RP; ++m) {
            double c[7];
#pragma unroll
            for (int d = 0; d < NT; ++d) c[d] = ro(S.coef + (size_t)d * S.npad + row0 + m * LANES);
            tmem_store<NT>(taddr + m * TMEM_ROW<NT>, c);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    // phase times of block 0 (thread 0), kept in shared memory
    __shared__ unsigned long long s_tp[6];
    const bool timing = prof != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
    if (timing) {
        for (int k = 0; k < 5; ++k) s_tp[k] = 0;
        s_tp[5] = global_ns();
    }
    auto mark = [&](int k) {
        if (timing) {
            const unsigned long long t = global_ns();
            s_tp[k] += t - s_tp[5];
            s_tp[5] = t;
        }
    };
    // row m of the thread
    auto row_product = [&](const KSys &S, int row, int m, const double *x) {
        if (RES && !far) return spmv_row_16<NT>(S, row, x, s_nbr + m * LANES, taddr + m * TMEM_ROW<NT>);
        return spmv_row_nb<NT>(S, row, x, S.nbr + row, (size_t)S.npad, taddr + m * TMEM_ROW<NT>);
    };
    // before a group adds to its chunk's lane sums: take them from the group
    // before it (named barrier 8 + gi: that group arrives, this one waits)
    auto take = [&](double &a, double &b) {
        if (PARTS > 1 && part > 0) {
            asm volatile("bar.sync %0, %1;" ::"r"(8 + gi), "n"(2 * LANES) : "memory");
            a = s_acc[gi - 1][0][lane];
            b = s_acc[gi - 1][1][lane];
        }
    };
    // afterwards: pass them on; true for the chunk's last group, which reduces them
    auto pass = [&](double a, double b) {
        if (PARTS > 1 && part < PARTS - 1) {
            s_acc[gi][0][lane] = a;
            s_acc[gi][1][lane] = b;
            asm volatile("bar.arrive %0, %1;" ::"r"(9 + gi), "n"(2 * LANES) : "memory");
            return false;
        }
        return true;
    };
    bool any = false;  // a launch that finds every system done returns at once
    for (int q = 0; q < A.nsys; ++q) any = any || state_active(sst[q]);
    if (!any) max_iters = 0;
    int it = 0;
    bool ok = true;
    for (; it < max_iters; ++it) {
        // K1: p = r + beta (p - w v); y = D^-1 p
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int r0 = (c - S.chunk_begin) * CH + lane0;
            const double beta = sst[si].beta, w = sst[si].w;
#pragma unroll
            for (int m0 = 0; m0 < RP; m0 += BATCH) {
                double v[BATCH], p[BATCH], r[BATCH], d[BATCH];
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    v[m] = S.v[row];
                    p[m] = S.p[row];
                    r[m] = S.r[row];
                    d[m] = ro(S.invdiag + row);
                }
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    const double pn = __fma_rn(beta, __fma_rn(-w, v[m], p[m]), r[m]);
                    S.p[row] = pn;
                    S.y[row] = d[m] * pn;
                }
            }
            if (RES) break;
        }
        if (!(ok = grid_sync(bar, target, &s_ok))) break;
        mark(0);
        // K2: v = A y, <r0, v>
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int lc = c - S.chunk_begin, r0 = lc * CH + lane0;
            double a = 0.0, none = 0.0;
            if constexpr (PARTS > 1) {
                double v[RP], q[RP];
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    const int row = r0 + m * LANES;
                    v[m] = row_product(S, row, m, S.y);
                    q[m] = S.r0[row];
                }
                take(a, none);
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    S.v[r0 + m * LANES] = v[m];
                    if (r0 + m * LANES < S.n) a = __fma_rn(q[m], v[m], a);
                }
            } else {
#pragma unroll kSpmvUnroll
                for (int m = 0; m < RP; ++m) {
                    const int row = r0 + m * LANES;
                    const double v = row_product(S, row, m, S.y);
                    S.v[row] = v;
                    if (row < S.n) a = __fma_rn(S.r0[row], v, a);
                }
            }
            if (pass(a, none)) {
                const double t = lanes_tree_sum(a, lane, sm[gi], gsync);
                if (lane == 0) S.part[4 * (size_t)S.nchunks + lc] = t;
            }
            if (RES) break;
        }
        if (!(ok = grid_sync(bar, target, &s_ok))) break;
        for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
            if (!state_active(sst[q])) continue;
            const KSys &S = A.sys[q];
            const double d = lanes_final_sum(S.part + 4 * (size_t)S.nchunks, S.nchunks, 1, lane, sm[gi], gsync);
            if (lane == 0) sst[q].alpha = sst[q].rho / d;
        }
        __syncthreads();
        mark(1);
        // K3: s = r - alpha v; z = D^-1 s
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int r0 = (c - S.chunk_begin) * CH + lane0;
            const double alpha = sst[si].alpha;
#pragma unroll
            for (int m0 = 0; m0 < RP; m0 += BATCH) {
                double v[BATCH], r[BATCH], d[BATCH];
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    v[m] = S.v[row];
                    r[m] = S.r[row];
                    d[m] = ro(S.invdiag + row);
                }
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    const double sv = __fma_rn(-alpha, v[m], r[m]);
                    S.s[row] = sv;
                    S.z[row] = d[m] * sv;
                }
            }
            if (RES) break;
        }
        if (!(ok = grid_sync(bar, target, &s_ok))) break;
        mark(2);
        // K4: t = A z, <t, t>, <t, s>
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int lc = c - S.chunk_begin, r0 = lc * CH + lane0;
            double att = 0.0, ats = 0.0;
            if constexpr (PARTS > 1) {
                double t[RP], q[RP];
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    const int row = r0 + m * LANES;
                    t[m] = row_product(S, row, m, S.z);
                    q[m] = S.s[row];
                }
                take(att, ats);
#pragma unroll
                for (int m = 0; m < RP; ++m) {
                    S.t[r0 + m * LANES] = t[m];
                    if (r0 + m * LANES < S.n) {
                        att = __fma_rn(t[m], t[m], att);
                        ats = __fma_rn(t[m], q[m], ats);
                    }
                }
            } else {
#pragma unroll kSpmvUnroll
                for (int m = 0; m < RP; ++m) {
                    const int row = r0 + m * LANES;
                    const double t = row_product(S, row, m, S.z);
                    S.t[row] = t;
                    if (row < S.n) {
                        att = __fma_rn(t, t, att);
                        ats = __fma_rn(t, S.s[row], ats);
                    }
                }
            }
            if (pass(att, ats)) {
                double tt, ts;
                lanes_tree_sum2(att, ats, lane, sm[gi], tt, ts, gsync);
                if (lane == 0) reinterpret_cast<double2 *>(S.part)[lc] = make_double2(tt, ts);
            }
            if (RES) break;
        }
        if (!(ok = grid_sync(bar, target, &s_ok))) break;
        for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
            if (!state_active(sst[q])) continue;
            const KSys &S = A.sys[q];
            double ftt, fts;
            lanes_final_sum2(S.part, S.nchunks, lane, sm[gi], ftt, fts, gsync);
            if (lane == 0) sst[q].w = (ftt > 0.0) ? fts / ftt : 0.0;
        }
        __syncthreads();
        mark(3);
        // K5: r = s - w t; <r0, r>, <r, r>
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int lc = c - S.chunk_begin, r0 = lc * CH + lane0;
            const double w = sst[si].w;
            double a0r = 0.0, arr = 0.0;
#pragma unroll
            for (int m0 = 0; m0 < RP; m0 += BATCH) {
                double t[BATCH], sv[BATCH], q[BATCH];
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    t[m] = S.t[row];
                    sv[m] = S.s[row];
                    q[m] = S.r0[row];
                }
                if (m0 == 0) take(a0r, arr);
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    const double r = __fma_rn(-w, t[m], sv[m]);
                    S.r[row] = r;
                    if (row < S.n) {
                        a0r = __fma_rn(q[m], r, a0r);
                        arr = __fma_rn(r, r, arr);
                    }
                }
            }
            if (pass(a0r, arr)) {
                double t0r, trr;
                lanes_tree_sum2(a0r, arr, lane, sm[gi], t0r, trr, gsync);
                if (lane == 0) reinterpret_cast<double2 *>(S.part + 2 * (size_t)S.nchunks)[lc] = make_double2(t0r, trr);
            }
            if (RES) break;
        }
        grid_arrive(bar, target);
        // x += alpha y + w z (no other block reads x)
        for (int c = cbegin; c < A.total_chunks; c += gstride) {
            const int si = sys_of_chunk(A, c);
            if (!state_active(sst[si])) continue;
            const KSys &S = A.sys[si];
            const int r0 = (c - S.chunk_begin) * CH + lane0;
            const double alpha = sst[si].alpha, w = sst[si].w;
#pragma unroll
            for (int m0 = 0; m0 < RP; m0 += BATCH) {
                double z[BATCH], y[BATCH], x[BATCH];
#pragma unroll
                for (int m = 0; m < BATCH; ++m) {
                    const int row = r0 + (m0 + m) * LANES;
                    z[m] = S.z[row];
                    y[m] = S.y[row];
                    x[m] = S.x[row];
                }
#pragma unroll
                for (int m = 0; m < BATCH; ++m)  // rows >= n of x are padding; they receive values computed from zeros
                    S.x[r0 + (m0 + m) * LANES] = __fma_rn(w, z[m], __fma_rn(alpha, y[m], x[m]));
            }
            if (RES) break;
        }
        if (!(ok = grid_wait(bar, target, &s_ok))) break;
        for (int q = gi; q < A.nsys; q += LOOP_GROUPS) {
            if (!state_active(sst[q])) continue;
            const KSys &S = A.sys[q];
            double f0r, frr;
            lanes_final_sum2(S.part + 2 * (size_t)S.nchunks, S.nchunks, lane, sm[gi], f0r, frr, gsync);
            if (lane == 0) {
                KState *st = &sst[q];
                st->rr = frr;
                st->iter += 1;
                st->work += 1;
                if (!(frr > st->tol2 && st->iter < st->maxit)) {
                    finish_loop(st);
                } else {
                    const double eps2 = DBL_EPSILON * DBL_EPSILON;
                    if (fabs(f0r) < eps2 * st->r0_sqnorm) {
                        st->paused = 1;  // the host recomputes r = b - A x and r0
                    } else {
                        st->beta = (f0r / st->rho) * (st->alpha / st->w);
                        st->rho = f0r;
                    }
                }
            }
        }
        __syncthreads();
        mark(4);
        bool any_active = false, any_paused = false;
        if constexpr (CAP <= KMAX) {
            for (int q = 0; q < A.nsys; ++q) {
                any_active = any_active || state_active(sst[q]);
                any_paused = any_paused || (sst[q].paused != 0 && sst[q].done == 0);
            }
        } else {  // the lanes of each warp split the systems
            for (int q = threadIdx.x & 31; q < A.nsys; q += 32) {
                any_active = any_active || state_active(sst[q]);
                any_paused = any_paused || (sst[q].paused != 0 && sst[q].done == 0);
            }
            any_active = __any_sync(0xffffffffu, any_active);
            any_paused = __any_sync(0xffffffffu, any_paused);
        }
        if (!any_active || any_paused) {
            ++it;
            break;
        }
    }
    if (RES) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_free(s_tmem);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < A.nsys) {
        KState k = sst[threadIdx.x];
        k.counter = 0;
        *A.sys[threadIdx.x].st = k;
    }
    if (timing) {
        for (int k = 0; k < 5; ++k) prof->ns[k] += s_tp[k];
        prof->iters += it;
        prof->ok = ok ? 1 : 0;
    }
}

// restart of paused systems: r = b - A x, r0 = r, rho = |r0|^2
template <int CAP, int G>
__global__ void __launch_bounds__(LANES *G, 8 / G) k_kr_restart(const __grid_constant__ KSetArgT<CAP> A) {
    __shared__ double sm[2 * CH + 8];
    __shared__ int sh[2];
    for (int c = blockIdx.x; c < A.total_chunks; c += gridDim.x) {
        const KSys &S = A.sys[sys_of_chunk(A, c)];
        if (!(__ldcg(&S.st->paused) != 0 && __ldcg(&S.st->done) == 0)) continue;
        const int lc = c - S.chunk_begin;
        chunk_residual<G, false>(S, lc, sm);
        if (arrive_last(S.st, (unsigned)S.nchunks, sh) && threadIdx.x < LANES) {
            const double rr = lanes_final_sum(S.part, S.nchunks, 2, threadIdx.x, sm + 2 * CH, GroupSync{1});
            if (threadIdx.x == 0) {
                KState *st = S.st;
                st->counter = 0;
                st->r0_sqnorm = rr;
                if (st->restarts++ == 0) st->iter = 0;
                st->beta = (rr / st->rho) * (st->alpha / st->w);
                st->rho = rr;
                st->paused = 0;
            }
        }
    }
}

#undef NS3D_CHUNK_LOOP

// y = A x for one system (tests and the residual checks of the drivers)
__global__ void __launch_bounds__(LANES) k_spmv(SysView A, const double *__restrict__ x, double *__restrict__ y) {
    KSys S;
    S.n = A.n;
    S.npad = A.npad;
    S.coef = A.coef;
    S.nbr = A.nbr;
    for (int c = blockIdx.x; c < A.nchunks; c += gridDim.x) {
        const int r0 = c * CH + threadIdx.x;
        st4(y + r0, spmv4(S, r0, x));
    }
}

// Test hook of the bounded grid barrier (ns3d_debug_barrier_timeout): while
// set, every loop-kernel launch's barrier waits for g_bar_bias arrivals that
// never come, for at most g_bar_limit_ns, then the launch ends with its
// error flag set.
static std::atomic<unsigned int> g_bar_bias{0};
static std::atomic<unsigned long long> g_bar_limit_ns{0};

void set_barrier_test(unsigned int bias, unsigned long long limit_ns) {
    g_bar_limit_ns = limit_ns;
    g_bar_bias = bias;
}

cudaError_t reset_grid_bar(GridBar *bar, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(GridBar), st);
    const unsigned int bias = g_bar_bias.load();
    if (e != cudaSuccess || bias == 0) return e;
    GridBar h;
    std::memset(&h, 0, sizeof h);
    h.bias = bias;
    h.limit_ns = g_bar_limit_ns.load();
    h.bias_others = bias > 1 ? 0 : bias;
    // pageable source: the copy is staged before the call returns
    return cudaMemcpyAsync(bar, &h, sizeof h, cudaMemcpyHostToDevice, st);
}

static std::atomic<int64_t> g_launches{0};
int64_t launch_count() { return g_launches.load(); }
void count_launches(int64_t n) { g_launches += n; }

static int g_sms = 0;
int device_sm_count() {
    if (g_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 152;
    }
    return g_sms;
}

// one block per chunk up to 32 blocks per SM (the hardware schedules the
// waves); beyond that, blocks walk the chunks grid-stride
static inline int kr_grid(int total_chunks) { return std::max(1, std::min(total_chunks, device_sm_count() * 32)); }

template <int CAP>
void launch_krylov_init(const KSetArgT<CAP> &A, cudaStream_t st) {
    if (A.total_chunks <= 0) return;
    count_launches(2);
    if (wide_chunks(A.total_chunks, device_sm_count()))
        k_kr_init<CAP, WIDE_G><<<kr_grid(A.total_chunks), LANES * WIDE_G, 0, st>>>(A);
    else
        k_kr_init<CAP, NARROW_G><<<kr_grid(A.total_chunks), LANES * NARROW_G, 0, st>>>(A);
    k_kr_init2<CAP><<<kr_grid(A.total_chunks), LANES, 0, st>>>(A);
}

// Blocks of a loop-kernel launch.  Every block must be resident at once
// (cooperative launch).  A solve that runs alone spreads its work units over
// every SM (one block per SM).  While k solves run in the process, a solve
// takes about 1/k of the SMs -- but at least one block per LOOP_GROUPS
// chunks of rows, so that no group holds more than one chunk per phase --
// and the loop kernels of concurrent solves, on their own streams, run side
// by side.
static std::atomic<int> g_active_solves{0};
ActiveSolve::ActiveSolve() { g_active_solves++; }
ActiveSolve::~ActiveSolve() { g_active_solves--; }
int active_solves() { return g_active_solves.load(); }

int loop_grid(int units, int units_per_chunk, int occ) {
    const int slots = device_sm_count() * std::max(occ, 1);
    const int active = std::max(1, g_active_solves.load());
    if (active == 1) return std::max(1, std::min(units, slots));
    // a fair share of the SMs, but never more than one chunk of rows per group
    const int per_block = LOOP_GROUPS * std::max(units_per_chunk, 1);
    const int dense = (units + per_block - 1) / per_block;
    const int fair = std::max(1, slots / active);
    return std::max(1, std::min(std::max(dense, std::min(fair, units)), slots));
}

// A merged set (the systems of many concurrent solves) spreads over its
// share of the SMs: all of them, or 1/share while `share` merged sets run.
template <int CAP>
static int krylov_loop_grid(int total_chunks, int occ, int share) {
    if (CAP > KMAX)
        return std::max(1, std::min(total_chunks, device_sm_count() * std::max(occ, 1) / std::max(share, 1)));
    return loop_grid(total_chunks, 1, occ);
}

// blocks the device can hold at once of the one-chunk kernel split over F blocks
template <int CAP, int F>
static int split_blocks() {
    static std::atomic<int> blocks{-1};
    int b = blocks.load();
    if (b >= 0) return b;
    b = 0;
    const void *fn = (const void *)k_kr_chunk<CAP, F>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkSmemBytes<F>) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(F);
        cfg.blockDim = dim3(kChunkRows<F>);
        cfg.dynamicSmemBytes = kChunkSmemBytes<F>;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = F;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess) b = n * F;
    }
    cudaGetLastError();
    blocks = b;
    return b;
}

// A set whose share of the SMs gives every chunk a block runs one chunk per
// block (krylov_chunk.cuh), a larger one several chunks per block: a block has
// one thread per row of its chunk, and the exchange needs every block
// resident.  While the share allows two or four blocks per chunk, a chunk is
// split over a cluster of them.  Measured, us per iteration, several per
// block -> one -> split: 5 chunks 35.4 -> 14.4 -> 12.5 (four blocks; 15.0 with
// two), 44 chunks 38.4 -> 17.5 -> 13.3 (two), 141 chunks 39.9 -> 19.3.
template <int CAP>
void plan_krylov(KSetArgT<CAP> &A, int share) {
    A.one_per_block = 0;
    const int n = A.total_chunks, sms = device_sm_count();
    if (n > sms || krylov_loop_grid<CAP>(n, 1, share) < n) return;
    const int avail = CAP > KMAX ? sms / std::max(share, 1) : sms / std::max(1, active_solves());
    if (4 * n <= std::min(avail, split_blocks<CAP, 4>())) A.one_per_block = 4;
    else if (2 * n <= std::min(avail, split_blocks<CAP, 2>())) A.one_per_block = 2;
    else A.one_per_block = 1;
}

template <int CAP, int F>
static cudaError_t launch_chunk(KSetArgT<CAP> &a, GridBar *bar, LoopProf *prof, int max_iters, cudaStream_t st) {
    void *args[] = {&a, &bar, &prof, &max_iters};
    return cudaLaunchCooperativeKernel((const void *)k_kr_chunk<CAP, F>, a.total_chunks * F, kChunkRows<F>, args,
                                       kChunkSmemBytes<F>, st);
}

template <int CAP>
cudaError_t launch_krylov_loop(const KSetArgT<CAP> &A, GridBar *bar, LoopProf *prof, int max_iters,
                               cudaStream_t st, int share) {
    if (A.total_chunks <= 0 || max_iters <= 0) return cudaSuccess;
    // the kernels in the order of their chunks per block; one block of 1024
    // threads per SM each
    struct Kernel {
        const void *fn;
        size_t smem;
        int chunks_per_block;  // at most (0: any number)
    };
    static const Kernel kernels[] = {{(const void *)k_kr_chunk<CAP, 1>, kChunkSmemBytes<1>, 1},
                                     {(const void *)k_kr_loop<CAP, 4>, kNbrSmemBytes<4>, LOOP_GROUPS / 4},
                                     {(const void *)k_kr_loop<CAP, 2>, kNbrSmemBytes<2>, LOOP_GROUPS / 2},
                                     {(const void *)k_kr_loop<CAP, 1>, kNbrSmemBytes<1>, LOOP_GROUPS},
                                     {(const void *)k_kr_loop<CAP, 0>, 0, 0}};
    static std::atomic<bool> ready{false};
    cudaError_t e = cudaSuccess;
    if (!ready.load()) {
        for (const Kernel &k : kernels) {
            if (k.smem) e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
            if (e != cudaSuccess) return e;
            int occ = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k.fn, LOOP_THREADS, k.smem);
            if (e != cudaSuccess) return e;
            if (occ <= 0) return cudaErrorLaunchOutOfResources;
        }
        ready = true;
    }
    e = reset_grid_bar(bar, st);
    if (e != cudaSuccess) return e;
    KSetArgT<CAP> a = A;
    void *args[] = {&a, &bar, &prof, &max_iters};
    count_launches(1);
    if (A.one_per_block == 4) return launch_chunk<CAP, 4>(a, bar, prof, max_iters, st);
    if (A.one_per_block == 2) return launch_chunk<CAP, 2>(a, bar, prof, max_iters, st);
    if (A.one_per_block == 1) return launch_chunk<CAP, 1>(a, bar, prof, max_iters, st);
    const int grid = krylov_loop_grid<CAP>(A.total_chunks, 1, share);
    int k = 1;
    while (kernels[k].chunks_per_block && A.total_chunks > grid * kernels[k].chunks_per_block) ++k;
    return cudaLaunchCooperativeKernel(kernels[k].fn, grid, LOOP_THREADS, args, kernels[k].smem, st);
}

template <int CAP>
void launch_krylov_restart(const KSetArgT<CAP> &A, cudaStream_t st) {
    if (A.total_chunks <= 0) return;
    count_launches(1);
    if (wide_chunks(A.total_chunks, device_sm_count()))
        k_kr_restart<CAP, WIDE_G><<<kr_grid(A.total_chunks), LANES * WIDE_G, 0, st>>>(A);
    else
        k_kr_restart<CAP, NARROW_G><<<kr_grid(A.total_chunks), LANES * NARROW_G, 0, st>>>(A);
}

// Loads the code of every kernel that a set of up to KMAX systems can run (CUDA
// loads a kernel when it is first used, and may allocate for it).
cudaError_t load_krylov_kernels() {
    for (const void *fn : {(const void *)k_kr_init<KMAX, WIDE_G>, (const void *)k_kr_init<KMAX, NARROW_G>,
                           (const void *)k_kr_init2<KMAX>, (const void *)k_kr_restart<KMAX, WIDE_G>,
                           (const void *)k_kr_restart<KMAX, NARROW_G>, (const void *)k_kr_chunk<KMAX, 1>,
                           (const void *)k_kr_chunk<KMAX, 2>, (const void *)k_kr_chunk<KMAX, 4>,
                           (const void *)k_kr_loop<KMAX, 0>, (const void *)k_kr_loop<KMAX, 1>,
                           (const void *)k_kr_loop<KMAX, 2>, (const void *)k_kr_loop<KMAX, 4>}) {
        cudaFuncAttributes at;
        const cudaError_t e = cudaFuncGetAttributes(&at, fn);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template void plan_krylov<KMAX>(KSetArg &, int);
template void plan_krylov<KMAX_MERGED>(KSetArgMerged &, int);
template void launch_krylov_init<KMAX>(const KSetArg &, cudaStream_t);
template void launch_krylov_init<KMAX_MERGED>(const KSetArgMerged &, cudaStream_t);
template cudaError_t launch_krylov_loop<KMAX>(const KSetArg &, GridBar *, LoopProf *, int, cudaStream_t, int);
template cudaError_t launch_krylov_loop<KMAX_MERGED>(const KSetArgMerged &, GridBar *, LoopProf *, int,
                                                     cudaStream_t, int);
template void launch_krylov_restart<KMAX>(const KSetArg &, cudaStream_t);
template void launch_krylov_restart<KMAX_MERGED>(const KSetArgMerged &, cudaStream_t);

void launch_spmv(const SysView &A, const double *x, double *y, cudaStream_t st) {
    if (A.n <= 0) return;
    count_launches(1);
    k_spmv<<<std::max(1, std::min(A.nchunks, device_sm_count() * 6)), LANES, 0, st>>>(A, x, y);
}

}  // namespace ns3d
