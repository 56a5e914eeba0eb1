// krylov_chunk.cuh -- the BiCGSTAB loop of small solve sets: one 1024-row
// chunk per block, one row per thread (included by krylov.cu).
//
// What bounds a small set is latency, not bytes: at 5 chunks an iteration of
// the group kernel (k_kr_loop) took 35 us, of which its 128 threads per chunk
// spent most waiting for their eight rows' loads in turn and in five grid
// barriers of 1.5 us.  Here
//   - the block keeps its chunk (coefficients, columns and vectors, 160 KB) in
//     shared memory for the whole launch; the only data that blocks exchange
//     are y, z and the chunk partials;
//   - the exchange needs no grid barrier.  Every exchanged double travels as
//     two 8-byte words that each hold 32 bits of it and the 32-bit epoch
//     (iteration number) it belongs to; a reader polls the words it needs
//     until both carry the epoch.  A word is valid by itself, so no fence is
//     needed: an all-reduce over the chunk partials takes 1.1-1.6 us instead
//     of barrier, fence and load (2.1 us), y and z reach a neighbouring block
//     in 1.3 us instead of 2.2 us;
//   - neighbours inside the chunk are read from shared memory;
//   - the systems of a set do not wait for each other.
// The arithmetic and its order are those of k_kr_loop: rows are multiplied by
// spmv_row's chain, lane l of a chunk accumulates rows l, l + 128, ... (the
// operands pass through shared memory), then the same trees.
//
// A word is rewritten only after every reader has read it: y of iteration
// i + 1 is stored after the reduction that ends iteration i, which needs a
// partial of every block of the system, stored after its last read of y.  The
// same holds for z and each partial.  The words start at zero (k_kr_init2)
// and the epoch, the system's iteration count of this solve, at 1.
//
// The words of y live in S.y (low halves) and S.s (high halves), those of z
// in S.z and S.t, those of the partials in S.part (chunk_tag_words).
//
// F > 1 (few chunks): a chunk's rows are split over the F blocks of a cluster,
// because a chunk alone keeps one SM's FP64 pipe (two operations per clock)
// busy for 5.8 us of an iteration while most SMs idle.  Each block hands the
// operands of the dot products to the cluster's first block, which accumulates
// them in the one order there is; every block combines the partials itself.
// They travel as asynchronous stores to that block's shared memory, counted by
// an mbarrier there, for which it alone waits (plain stores and a barrier of
// the cluster made every block wait: 14.4 instead of 13.3 us at 44 chunks).
// The operands of a reduction overwrite those of the one before, which the
// first block has accumulated: its partial is part of the scalar that every
// block needed to get there.  So no block is ever more than one hand-over
// ahead of the first one, also when waits run out.
//
// What bounds it now: per block and iteration 27 FP64 operations a row at two
// per clock (6.7 us for a whole chunk), three reductions of about 2.3 us (a chain of eight
// 68-cycle FMAs, two trees, one exchange, one division) and two exchanges of
// y and z.
#pragma once

#include <algorithm>

#include "tags.cuh"

namespace ns3d {

// S.part of a system: [0, 4 n) the plain partials of k_kr_init and
// k_kr_restart, then 2 words per kind and chunk
__device__ __forceinline__ unsigned long long *chunk_tag_words(const KSys &S) {
    return reinterpret_cast<unsigned long long *>(S.part + 4 * (size_t)S.nchunks);
}
static_assert(PART_PER_CHUNK >= 4 + 2 * TAG_KINDS, "tagged partials");

// rows of a block; shared memory: its rows' data and, for a split chunk, the
// chunk's r0 and two operands (at least 120 KB, so that an SM takes one block)
template <int F>
constexpr int kChunkRows = CH / F;
template <int F>
constexpr size_t kChunkSmemBytes =
    F == 1 ? (size_t)CH * (17 * sizeof(double) + 6 * sizeof(int))
           : std::max((size_t)120 << 10,
                      kChunkRows<F> * (17 * sizeof(double) + 6 * sizeof(int)) + (size_t)3 * CH * sizeof(double));

// An mbarrier in the first block counts the bytes that have arrived.
__device__ __forceinline__ unsigned int smem_addr(const void *p) { return (unsigned int)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *m) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;\n fence.mbarrier_init.release.cluster;" ::"r"(smem_addr(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *m, unsigned int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(m)), "r"(bytes) : "memory");
}
// bytes that will not arrive count as arrived
__device__ __forceinline__ void mbar_forgo(unsigned long long *m, unsigned int bytes) {
    asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(m)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_done(unsigned long long *m, unsigned int parity) {
    unsigned int ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(m)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// v to p, an address in this block's shared memory, in the cluster's first
// block: counted by the barrier m there, or ordered by the next cluster barrier
__device__ __forceinline__ void store_first(double *p, double v, unsigned long long *m) {
    unsigned int a, b;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_addr(p)));
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(b) : "r"(smem_addr(m)));
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(b)
                 : "memory");
}
__device__ __forceinline__ void store_first(unsigned int *p, unsigned int v) {
    unsigned int a;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_addr(p)));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// The column values of the thread's row, slots W, E, S, N, B, T: neighbours
// in the block's rows from `own` (shared), the others from their tagged words; a
// missing neighbour gets the row's own value (its product is skipped).
// Outside the block a row has W and E and, at the block's ends, one of S and
// N and one of B and T: those four are polled at once (a second round trip
// costs 0.6 us; polling all six at once needs registers that spill).
template <int ROWS>
__device__ __forceinline__ void gather_tagged(const int *s_col, int base, int t, const double *own, const double *lo,
                                              const double *hi, unsigned int ep, double (&x)[6], GridBar *bar,
                                              int &bad) {
    unsigned int need = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int c = s_col[d * ROWS];
        const unsigned int q = (unsigned int)(c - base);
        const bool ext = c >= 0 && q >= (unsigned int)ROWS;
        x[d] = own[!ext && c >= 0 ? q : t];
        need |= (unsigned int)ext << d;
    }
    PollLimit limit(bar, bad);
    while (need) {
        const bool north = (need >> 2 & 1u) == 0, top = (need >> 4 & 1u) == 0;
        const unsigned int bit[4] = {need & 1u, need & 2u, need & (north ? 8u : 4u), need & (top ? 32u : 16u)};
        const int slot[4] = {0, 1, north ? 3 : 2, top ? 5 : 4};
        unsigned long long a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (bit[k]) {
                const int c = s_col[slot[k] * ROWS];
                a[k] = ld_word(lo + c);
                b[k] = ld_word(hi + c);
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (bit[k] && tag_ok(a[k], b[k], ep)) {
                const double val = tag_value(a[k], b[k]);
                if (k < 2) x[k] = val;
                else if (k == 2) (north ? x[3] : x[2]) = val;
                else (top ? x[5] : x[4]) = val;
                need &= ~bit[k];
            }
        if (need && !limit.again()) return;
    }
}

// One dot product of a system over all its chunks, by one group of 128
// threads: with `mine` (the block that has the chunk's operands) the chunk's
// partial, published; then the sum of all chunks' partials in the fixed order.
// Valid in the group's first thread.  Every thread of the group calls
// `published` once its part in publishing is done.
template <class Published>
__device__ __forceinline__ double dot_all(const KSys &S, int lc, int kind, bool mine, const double *a, const double *b,
                                          int lane, unsigned int ep, unsigned int want, double *red, GroupSync sync,
                                          GridBar *bar, int &bad, Published published) {
    const int n = S.nchunks;
    unsigned long long *slots = chunk_tag_words(S) + 2 * (size_t)kind * n;
    unsigned int *counter = tag_counter(S.part, n, kind);
    if (mine) {
        const double part = group_tree(lane_dot(a, b, lane, min(CH, S.n - lc * CH)), LANES, lane, red, sync);
        if (lane == 0) {
            st_words(slots + 2 * (size_t)lc, tag_lo(part, ep), tag_hi(part, ep));
            if (n > 32) count_arrival(counter);
        }
    }
    published();
    if (n <= 32 && lane >= 32) return 0.0;  // the first warp alone combines them
    PollLimit limit(bar, bad);
    if (n > 32) {  // fewer words are polled directly: one round trip less, and one warp only
        if (lane == 0) wait_arrivals(counter, ep * (unsigned int)n, limit);
        sync();
    }
    double sum = 0.0;
    for (int i = lane; i < n; i += LANES) {
        unsigned long long lo, hi;
        while (true) {
            ld_words(slots + 2 * (size_t)i, lo, hi);
            if (tag_ok(lo, hi, want) || !limit.again()) break;
        }
        sum = sum + tag_value(lo, hi);
    }
    return group_tree(sum, min(n, LANES), lane, red + LANES / 32, sync);
}

// (The cluster's size is part of the kernel: as an attribute of a cooperative
// launch it made the launch fail under a profiler.)
template <int CAP, int F>
__global__ void __cluster_dims__(F, 1, 1) __launch_bounds__(kChunkRows<F>, 1)
    k_kr_chunk(const __grid_constant__ KSetArgT<CAP> A, GridBar *bar, LoopProf *prof, int max_iters) {
    static_assert(CH == 1024, "one thread per row of a chunk");
    extern __shared__ double sm_chunk[];
    constexpr int RB = kChunkRows<F>;
    // the block's rows: coefficients and vectors, [7 + 10][RB]
    double *const s_cf = sm_chunk;
    double *const s_r0 = s_cf + 7 * RB, *const s_x = s_r0 + RB, *const s_p = s_x + RB, *const s_y = s_p + RB,
                  *const s_v = s_y + RB, *const s_s = s_v + RB, *const s_z = s_s + RB, *const s_t = s_z + RB,
                  *const s_r = s_t + RB, *const s_invd = s_r + RB;
    int *const s_col = reinterpret_cast<int *>(s_invd + RB) + threadIdx.x;  // [6][RB]: the thread's columns
    // the chunk's r0 and operands of the dot products (in the cluster's first block)
    double *const o_r0 = F == 1 ? s_r0 : reinterpret_cast<double *>(s_col - threadIdx.x + 6 * RB);
    double *const o_a = o_r0 + CH, *const o_b = o_a + CH;  // F > 1
    __shared__ KState st;
    __shared__ double s_red[2][2 * (LANES / 32)], s_other, s_ratio;
    __shared__ __align__(8) unsigned long long s_handed;  // in the cluster's first block
    __shared__ unsigned int s_sent[F];                    // there too
    const int t = threadIdx.x, gi = t / LANES;
    const int chunk = (int)blockIdx.x / F, part = (int)blockIdx.x % F;
    const KSys &S = A.sys[sys_of_chunk(A, chunk)];
    const int lc = chunk - S.chunk_begin, base = lc * CH + part * RB, row = base + t;
    const bool first = part == 0;
    if (t == 0) {
        st = *S.st;
        if (F > 1) mbar_init(&s_handed);
    }
    const bool timing = prof != nullptr && blockIdx.x == 0 && t == 0;
    __shared__ unsigned long long s_tp[6];  // phase times of block 0
    if (timing)
        for (int k = 0; k < 6; ++k) s_tp[k] = 0;
    __syncthreads();
    if (!state_active(st)) return;  // the same in every block of the system
    bool has[6];  // the row's entries
    {
        const size_t np = (size_t)S.npad;
#pragma unroll
        for (int d = 0; d < 7; ++d) s_cf[d * RB + t] = ro(S.coef + d * np + row);
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            const int c = ro(S.nbr + d * np + row);
            s_col[d * RB] = c;
            has[d] = c >= 0;
        }
    }
    if (F == 1) s_r0[t] = S.r0[row];
    else if (first)
        for (int q = t; q < CH; q += RB) o_r0[q] = S.r0[lc * CH + q];
    s_invd[t] = ro(S.invdiag + row);
    s_p[t] = S.p[row];
    s_v[t] = S.v[row];
    s_r[t] = S.r[row];
    s_x[t] = S.x[row];
    const bool wlate = has[0] && s_col[0] == row - 1, eearly = has[1] && s_col[RB] == row + 1;
    const bool rare = __any_sync(0xffffffffu, wlate || eearly);
    // A x for the thread's row from its own value and the six columns'; the
    // chain of spmv_row_nb
    auto product = [&](double xp, const double (&xc)[6]) {
        const double *cf = s_cf + t;
        double acc = 0.0;
        if (rare) {
            if (!wlate && has[0]) acc = __fma_rn(cf[1 * RB], xc[0], acc);
            if (has[2]) acc = __fma_rn(cf[3 * RB], xc[2], acc);
            if (has[4]) acc = __fma_rn(cf[5 * RB], xc[4], acc);
            if (wlate) acc = __fma_rn(cf[1 * RB], xc[0], acc);
            acc = __fma_rn(cf[0], xp, acc);
            if (eearly) acc = __fma_rn(cf[2 * RB], xc[1], acc);
            if (has[5]) acc = __fma_rn(cf[6 * RB], xc[5], acc);
            if (has[3]) acc = __fma_rn(cf[4 * RB], xc[3], acc);
            if (!eearly && has[1]) acc = __fma_rn(cf[2 * RB], xc[1], acc);
        } else {
            if (has[0]) acc = __fma_rn(cf[1 * RB], xc[0], acc);
            if (has[2]) acc = __fma_rn(cf[3 * RB], xc[2], acc);
            if (has[4]) acc = __fma_rn(cf[5 * RB], xc[4], acc);
            acc = __fma_rn(cf[0], xp, acc);
            if (has[5]) acc = __fma_rn(cf[6 * RB], xc[5], acc);
            if (has[3]) acc = __fma_rn(cf[4 * RB], xc[3], acc);
            if (has[1]) acc = __fma_rn(cf[2 * RB], xc[1], acc);
        }
        return acc;
    };
    auto mark = [&](int k) {
        if (timing) {
            const unsigned long long now = global_ns();
            s_tp[k] += now - s_tp[5];
            s_tp[5] = now;
        }
    };
    if (timing) s_tp[5] = global_ns();
    // a test (ns3d_debug_barrier_timeout) makes every wait for a chunk partial
    // run out, or those of the clusters' first blocks: it waits for epochs that
    // are never written
    // (read through one pointer: a choice between two conditions took 1% of an
    // iteration)
    const unsigned int *const hook = first ? &bar->bias : &bar->bias_others;
    const unsigned int never = __ldcg(hook) ? 0x80000000u : 0u;
    const GroupSync sync{gi + 1};
    auto nothing = [] {};
    // the operands of a dot product (`count` a row) are complete where it is
    // accumulated; false when a wait ran out
    int bad = 0;
    unsigned int parity = 0;
    bool late = false;  // the wait for the operands ran out
    // in the iteration that ends the loop because a wait ran out: operands a
    // row that the block has handed over, and that the first block has got
    unsigned int sent = 0, taken = 0;
    auto handed = [&](unsigned int count) {
        if (F > 1 && first) {
            if (t == 0) mbar_expect(&s_handed, count * CH * (unsigned int)sizeof(double));
            PollLimit limit(bar, bad);
            bool done;
            while (!(done = mbar_done(&s_handed, parity)) && limit.again()) {
            }
            if (done) parity ^= 1u;
            else late = true;
        }
        return __syncthreads_or(bad) == 0;
    };
    auto gave_up = [&](unsigned int before, unsigned int after) {
        sent = after;
        taken = late ? before : after;
    };
    if (F > 1) cluster_barrier();  // every block of the cluster runs
    int it = 0;
    for (; it < max_iters; ++it) {
        const unsigned int ep = (unsigned int)st.work + 1u;  // uniform: st changes only between block barriers
        double xc[6];
        // K1: p = r + beta (p - w v); y = D^-1 p
        {
            const double p = __fma_rn(st.beta, __fma_rn(-st.w, s_v[t], s_p[t]), s_r[t]);
            const double y = s_invd[t] * p;
            st_word(S.y + row, tag_lo(y, ep));
            st_word(S.s + row, tag_hi(y, ep));
            s_y[t] = y;
            s_p[t] = p;
        }
        __syncthreads();
        mark(0);
        // K2: v = A y, <r0, v>
        gather_tagged<RB>(s_col, base, t, s_y, S.y, S.s, ep, xc, bar, bad);
        {
            const double v = product(s_y[t], xc);
            s_v[t] = v;
            if (F > 1) store_first(o_a + part * RB + t, v, &s_handed);
        }
        if (!handed(1)) {
            gave_up(0, 1);
            break;
        }
        if (gi == 0) {
            const double d = dot_all(S, lc, 0, first, o_r0, F == 1 ? s_v : o_a, t, ep, ep | never, s_red[0], sync, bar, bad,
                                     nothing);
            if (t == 0) st.alpha = st.rho / d;
        }
        if (__syncthreads_or(bad)) {
            gave_up(0, 1);
            break;
        }
        mark(1);
        // K3: s = r - alpha v; z = D^-1 s
        {
            const double s = __fma_rn(-st.alpha, s_v[t], s_r[t]);
            const double z = s_invd[t] * s;
            st_word(S.z + row, tag_lo(z, ep));
            st_word(S.t + row, tag_hi(z, ep));
            s_z[t] = z;
            s_s[t] = s;
        }
        __syncthreads();
        mark(2);
        // K4: t = A z, <t, t>, <t, s>
        gather_tagged<RB>(s_col, base, t, s_z, S.z, S.t, ep, xc, bar, bad);
        {
            const double tv = product(s_z[t], xc);
            s_t[t] = tv;
            if (F > 1) {
                store_first(o_a + part * RB + t, tv, &s_handed);
                store_first(o_b + part * RB + t, s_s[t], &s_handed);
            }
        }
        if (!handed(2)) {
            gave_up(1, 3);
            break;
        }
        if (gi < 2) {
            const double *ot = F == 1 ? s_t : o_a, *os = F == 1 ? s_s : o_b;
            const double d = dot_all(S, lc, 1 + gi, first, ot, gi == 0 ? ot : os, t % LANES, ep, ep | never, s_red[gi],
                                     sync, bar, bad, nothing);
            if (t == LANES) s_other = d;
            asm volatile("bar.sync 3, %0;" ::"n"(2 * LANES) : "memory");
            if (t == 0) st.w = (d > 0.0) ? s_other / d : 0.0;
        }
        if (__syncthreads_or(bad)) {
            gave_up(1, 3);
            break;
        }
        mark(3);
        // K5: r = s - w t, <r0, r>, <r, r>; x += alpha y + w z
        const double alpha = st.alpha, w = st.w;
        {
            const double r = __fma_rn(-w, s_t[t], s_s[t]);
            s_r[t] = r;
            if (F > 1) store_first(o_a + part * RB + t, r, &s_handed);
        }
        if (!handed(1)) {
            gave_up(3, 4);
            break;
        }
        // x and the second ratio of beta in the time the partials travel: before
        // they are published this FP64 work would delay them
        auto update_x = [&](int q) { s_x[q] = __fma_rn(w, s_z[q], __fma_rn(alpha, s_y[q], s_x[q])); };
        auto ratio = [&](int by) {  // by the warp of thread `by`
            if (t / 32 != by / 32) return;
            if (t == by) s_ratio = alpha / w;
            asm volatile("bar.arrive 5, 64;" ::: "memory");
        };
        if (gi < 2) {
            auto published = [&] {
                if (F == 1) {  // the other warps may start
                    asm volatile("bar.arrive 4, %0;" ::"n"(CH) : "memory");
                } else {  // not the groups' first warps: they go on to the partials
                    ratio(96);
                    if (t / 32 % 4 != 0) update_x(t);
                    if (t / 32 % 4 == 1) update_x(t - 32);
                }
            };
            const double *orr = F == 1 ? s_r : o_a;
            const double d = dot_all(S, lc, 3 + gi, first, gi == 0 ? o_r0 : orr, orr, t % LANES, ep, ep | never, s_red[gi],
                                     sync, bar, bad, published);
            if (t == LANES) s_other = d;
            asm volatile("bar.sync 3, %0;" ::"n"(2 * LANES) : "memory");
            if (t < 32) asm volatile("bar.sync 5, 64;" ::: "memory");  // s_ratio is written
            if (t == 0) {
                const double f0r = d, frr = s_other;
                st.rr = frr;
                st.iter += 1;
                st.work += 1;
                if (!(frr > st.tol2 && st.iter < st.maxit)) {
                    finish_loop(&st);
                } else if (fabs(f0r) < DBL_EPSILON * DBL_EPSILON * st.r0_sqnorm) {
                    st.paused = 1;  // the host recomputes r = b - A x and r0
                } else {
                    st.beta = (f0r / st.rho) * s_ratio;
                    st.rho = f0r;
                }
            }
        } else {
            if (F == 1) {
                ratio(2 * LANES);
                asm volatile("bar.sync 4, %0;" ::"n"(CH) : "memory");
                for (int q = t - 2 * LANES; q < CH; q += CH - 2 * LANES) update_x(q);
            } else {
                update_x(t);
            }
        }
        if (__syncthreads_or(bad)) {
            gave_up(3, 4);
            break;
        }
        mark(4);
        if (!state_active(st)) {
            ++it;
            break;
        }
    }
    S.p[row] = s_p[t];
    S.v[row] = s_v[t];
    S.r[row] = s_r[t];
    S.x[row] = s_x[t];
    if (lc == 0 && part == 0 && t == 0) {
        st.counter = 0;
        *S.st = st;
    }
    if (timing) {
        for (int k = 0; k < 5; ++k) prof->ns[k] += s_tp[k];
        prof->iters += it;
        prof->ok = bad ? 0 : 1;
    }
    // The first block's shared memory stays until the last store to it has
    // arrived.  At a regular end it has waited for all of them.  When a wait
    // ran out, operands may be on their way that it did not wait for: of a
    // hand-over whose wait ran out there (the barrier expects all blocks'
    // bytes, some may never have been sent), or of the one after its last (its
    // wait for the partials ran out, another block's did not; the barrier
    // expects nothing).  Every block stores the operands of all its rows or of
    // none, so the blocks' counts say what is still to come; it is waited for
    // before the block ends.
    if (F > 1) {
        if (t == 0) store_first(&s_sent[part], 4u * it + sent);
        cluster_barrier();
        if (first && t == 0) {
            unsigned int open = 0;
#pragma unroll
            for (int q = 0; q < F; ++q) open += s_sent[q] - (4u * it + taken);
            if (open > 0) {
                constexpr unsigned int bytes = RB * sizeof(double);
                if (sent == taken) mbar_expect(&s_handed, open * bytes);
                else if (open < (sent - taken) * F) mbar_forgo(&s_handed, ((sent - taken) * F - open) * bytes);
                PollLimit limit(bar, bad);
                while (!mbar_done(&s_handed, parity) && limit.again()) {
                }
            }
        }
    }
}

}  // namespace ns3d
