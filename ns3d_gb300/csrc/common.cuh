// common.cuh -- shared definitions of the NS3D GB300 kernels.
//
// Floating-point contract (every FP64 translation unit is compiled with
// --fmad=false): expressions round exactly as written, and fused
// multiply-adds appear only where __fma_rn is called.  Together with the
// fixed reduction order below this makes the device results reproducible
// run to run and identical to the CPU restatement used by the tests.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ns3d {

// ---- fixed-order reductions ---------------------------------------------
// Rows are cut into chunks of CH = 1024.  A chunk is processed by one block
// of LANES = 128 threads; thread (lane) l owns rows l, l+128, ..., l+896 of
// the chunk (coalesced) and accumulates them in that order.  Each warp's 32
// lane values are combined by a halving tree (offsets 16, 8, 4, 2, 1), then
// the 4 warp sums by a halving tree (offsets 2, 1).  Chunk partials of one
// system are combined the same way by the last block to finish: lane l sums
// partials l, l+128, ... in order, then the trees.
constexpr int LANES = 128;
constexpr int RPL = 8;
constexpr int CH = LANES * RPL;

__device__ __forceinline__ double warp_tree_sum(double v) {
    // offsets 16..1 of the halving tree inside one warp; lane 0 ends with the
    // value the tree assigns to position 0 of this warp's 32-lane group
    v = v + __shfl_down_sync(0xffffffffu, v, 16);
    v = v + __shfl_down_sync(0xffffffffu, v, 8);
    v = v + __shfl_down_sync(0xffffffffu, v, 4);
    v = v + __shfl_down_sync(0xffffffffu, v, 2);
    v = v + __shfl_down_sync(0xffffffffu, v, 1);
    return v;
}

// Tree sum over LANES threads (lane = this thread's index among them) that
// synchronize with `sync`, the named barrier of their group.  Returns the tree
// sum in lane 0 (other lanes get an unspecified value).  `sm` needs one value
// per warp.
template <class T, class Sync>
__device__ __forceinline__ T lanes_tree_sum(T v, int lane, T *sm, Sync sync) {
    v = v + __shfl_down_sync(0xffffffffu, v, 16);
    v = v + __shfl_down_sync(0xffffffffu, v, 8);
    v = v + __shfl_down_sync(0xffffffffu, v, 4);
    v = v + __shfl_down_sync(0xffffffffu, v, 2);
    v = v + __shfl_down_sync(0xffffffffu, v, 1);
    if ((lane & 31) == 0) sm[lane >> 5] = v;
    sync();
    T r = T(0);
    if (lane < 32) {
        r = (lane < LANES / 32) ? sm[lane] : T(0);
        for (int off = LANES / 64; off >= 1; off >>= 1) r = r + __shfl_down_sync(0xffffffffu, r, off);
    }
    sync();
    return r;
}

// Two tree sums at once, each with exactly the pairings of lanes_tree_sum.
// After the first level of a warp, lanes 0-15 carry the first sum and lanes
// 16-31 the second, so every later level is one shuffle and one add for
// both (FP64 issue is scarce on this GPU).  Results valid in lane 0.  `sm`
// needs two values per warp.
template <class T, class Sync>
__device__ __forceinline__ void lanes_tree_sum2(T a, T b, int lane, T *sm, T &ra, T &rb, Sync sync) {
    static_assert(2 * (LANES / 32) <= 32, "warp sums of both trees fit one warp");
    ra = T(0);
    rb = T(0);
    const bool lo = (lane & 16) == 0;
    // offset 16: lane l < 16 forms a_l + a_(l+16), lane l >= 16 forms b_(l-16) + b_l
    T v = (lo ? a : b) + __shfl_xor_sync(0xffffffffu, lo ? b : a, 16);
    v = v + __shfl_down_sync(0xffffffffu, v, 8);
    v = v + __shfl_down_sync(0xffffffffu, v, 4);
    v = v + __shfl_down_sync(0xffffffffu, v, 2);
    v = v + __shfl_down_sync(0xffffffffu, v, 1);
    constexpr int NW = LANES / 32;
    if ((lane & 31) == 0) sm[lane >> 5] = v;
    if ((lane & 31) == 16) sm[NW + (lane >> 5)] = v;
    sync();
    if (lane < 32) {
        T r = (lane < 2 * NW) ? sm[lane] : T(0);
        for (int off = NW / 2; off >= 1; off >>= 1) r = r + __shfl_down_sync(0xffffffffu, r, off);
        const T r2 = __shfl_sync(0xffffffffu, r, NW);
        ra = r;
        rb = r2;
    }
    sync();
}

// named barrier `id` (1..15) over the LANES threads of one group
struct GroupSync {
    int id;
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(LANES) : "memory");
    }
};

__device__ __forceinline__ double dmaxv(double a, double b) { return (b > a) ? b : a; }
__device__ __forceinline__ double dminv(double a, double b) { return (b < a) ? b : a; }

// maximum / minimum over the LANES threads of a group (exact in any order);
// valid in every thread.  sm: LANES / 32 doubles.
template <bool MAX, class Sync>
__device__ __forceinline__ double lanes_extreme(double v, int lane, double *sm, Sync sync) {
    for (int off = 16; off >= 1; off >>= 1) {
        const double o = __shfl_down_sync(0xffffffffu, v, off);
        v = MAX ? dmaxv(v, o) : dminv(v, o);
    }
    if ((lane & 31) == 0) sm[lane >> 5] = v;
    sync();
    double r = sm[0];
    for (int w = 1; w < LANES / 32; ++w) r = MAX ? dmaxv(r, sm[w]) : dminv(r, sm[w]);
    sync();
    return r;
}

// ---- chunk kernels ----------------------------------------------------------
// The kernels that compute per-row operands and reduce them run one chunk per
// block of LANES * G threads: thread (g, lane) computes rows
// lane + LANES m, m in [g RPL / G, (g + 1) RPL / G), the operands pass through
// shared memory, and group j accumulates sum j lane by lane in the fixed
// order.  A row costs several dependent loads, so a small system is bound by
// the latency of the rows a thread walks in turn: with one group these
// kernels took 19 us (k_kr_init), 38 (k_dc_resid), 40 (k_dc_step) and 61-72 us
// (k_divergence) whatever the size, with eight 11, 17, 21 and 24 us.  Above
// WIDE_CHUNKS_PER_SM chunks per SM the other blocks cover that latency and a
// wide block only waits for its own reduction (10.5 M rows: k_dc_resid 426 us
// with eight groups, 287 with two).  The launch bounds ask for 1024 threads per
// SM in either form, so 64 registers a thread: k_kr_init, k_kr_restart,
// k_dc_resid and k_dc_step with two groups spill 110 to 200 bytes a thread.
constexpr int WIDE_CHUNKS_PER_SM = 2;
constexpr int WIDE_G = 8, NARROW_G = 2;
inline bool wide_chunks(int nchunks, int sms) { return nchunks <= WIDE_CHUNKS_PER_SM * sms; }

// a lane's accumulation of sum a[q] b[q] over its rows of a chunk, from the
// operands in shared memory (rows: rows of the chunk below the system's n)
__device__ __forceinline__ double lane_dot(const double *a, const double *b, int lane, int rows) {
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < RPL; ++m)
        if (lane + m * LANES < rows) acc = __fma_rn(a[lane + m * LANES], b[lane + m * LANES], acc);
    return acc;
}

// Final combination of `n` chunk partials (strided by `stride` doubles):
// lane l sums partials l, l+LANES, ... in order, then the halving tree.
// Result valid in lane 0.
// The partials a lane adds are loaded 8 at a time before they are added (in
// the same order), so the sum waits for one L2 round trip per 8 partials
// instead of one per partial.
constexpr int FINAL_BATCH = 8;

template <int BATCH = FINAL_BATCH, class Sync>
__device__ __forceinline__ double lanes_final_sum(const double *part, int n, int stride, int lane, double *sm,
                                                  Sync sync) {
    double a = 0.0;
    for (int base = lane; base < n; base += BATCH * LANES) {
        double v[BATCH];
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
            const int i = base + k * LANES;
            v[k] = (i < n) ? __ldcg(part + (size_t)i * stride) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < BATCH; ++k)
            if (base + k * LANES < n) a = a + v[k];
    }
    return lanes_tree_sum<double>(a, lane, sm, sync);
}
// the same for the interleaved pairs part[2i] and part[2i+1] (16-byte aligned)
template <class Sync>
__device__ __forceinline__ void lanes_final_sum2(const double *part, int n, int lane, double *sm, double &ra,
                                                 double &rb, Sync sync) {
    double a = 0.0, b = 0.0;
    for (int base = lane; base < n; base += FINAL_BATCH * LANES) {
        double2 v[FINAL_BATCH];
#pragma unroll
        for (int k = 0; k < FINAL_BATCH; ++k) {
            const int i = base + k * LANES;
            v[k] = (i < n) ? __ldcg(reinterpret_cast<const double2 *>(part) + i) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int k = 0; k < FINAL_BATCH; ++k)
            if (base + k * LANES < n) {
                a = a + v[k].x;
                b = b + v[k].y;
            }
    }
    lanes_tree_sum2<double>(a, b, lane, sm, ra, rb, sync);
}

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace ns3d
