// tags.cuh -- what the loop kernels with resident chunks (krylov_chunk.cuh,
// mixed_chunk.cuh) share: 8-byte words that carry 32 bits of data and the
// 32-bit epoch it belongs to, bounded polling, and their reduction tree.
#pragma once

#include "loop.cuh"

namespace ns3d {

constexpr int TAG_KINDS = 5;  // <r0,v>, <t,t>, <t,s>, <r0,r>, <r,r>
// One arrival counter per kind, each on its own 128-byte line, behind the
// partials of a system (PART_FIXED doubles beyond PART_PER_CHUNK a chunk).
// A reader first waits, with one thread, until the counter says that every
// block has stored its partial, then reads the words: the counter orders
// nothing (relaxed, no fence; a word that is not there yet is read again), it
// keeps 128 threads of every block from polling the same lines.  All-reduce
// over 141 blocks: 1.6 us; 2.5 us polling the words alone, 2.0 us with eight
// copies of them; 2.1 us with a barrier, fence and load.
__device__ __forceinline__ unsigned int *tag_counter(double *part, int nchunks, int kind) {
    return reinterpret_cast<unsigned int *>(part + ((size_t)PART_PER_CHUNK * nchunks + 15) / 16 * 16 + 16 * kind);
}
static_assert(PART_FIXED >= 16 + 16 * TAG_KINDS, "arrival counters");

__device__ __forceinline__ unsigned long long tag_lo(double v, unsigned int ep) {
    return ((unsigned long long)ep << 32) | (unsigned int)__double2loint(v);
}
__device__ __forceinline__ unsigned long long tag_hi(double v, unsigned int ep) {
    return ((unsigned long long)ep << 32) | (unsigned int)__double2hiint(v);
}
__device__ __forceinline__ double tag_value(unsigned long long lo, unsigned long long hi) {
    return __hiloint2double((int)(unsigned int)hi, (int)(unsigned int)lo);
}
__device__ __forceinline__ bool tag_ok(unsigned long long lo, unsigned long long hi, unsigned int ep) {
    return (unsigned int)(lo >> 32) == ep && (unsigned int)(hi >> 32) == ep;
}
__device__ __forceinline__ unsigned long long ld_word(const void *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(void *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void ld_words(const void *p, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_words(void *p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}

// Bounded polling: false when the wait has run out (the same limit as the
// grid barrier's), after setting bar->err and the thread's flag; the block
// stops at its next barrier, which combines the flags.
struct PollLimit {
    GridBar *bar;
    int &bad;
    unsigned int polls = 0;
    unsigned long long t0 = 0;
    __device__ PollLimit(GridBar *b, int &f) : bar(b), bad(f) {}
    __device__ __forceinline__ bool again() {
        if ((++polls & 255u) != 0) return true;
        const unsigned long long now = global_ns();
        if (polls == 256u) t0 = now;
        const unsigned long long lim = bar->limit_ns ? bar->limit_ns : kBarrierLimitNs;
        if (now - t0 <= lim && polls <= 0x7fffffffu) return true;
        atomicExch(&bar->err, 1);
        bad = 1;
        return false;
    }
};

__device__ __forceinline__ void count_arrival(unsigned int *c) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
}
// by one thread: until `target` arrivals (the counters only grow)
__device__ __forceinline__ void wait_arrivals(const unsigned int *c, unsigned int target, PollLimit &limit) {
    unsigned int v;
    do {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
    } while ((int)(v - target) < 0 && limit.again());
}

// The tree sum of lanes_tree_sum over the 128 threads of one group, of which
// only the first `n` hold a value and the others +0: a level that would only
// add those zeros is left out (v + 0 = v; no value here is -0).  FP64 adds
// have a latency of 68 cycles, a level with its shuffle 94.  Valid in the
// group's first thread; with n <= 32 only its first warp takes part.
__device__ __forceinline__ double group_tree(double v, int n, int lane, double *red, GroupSync sync) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
        if (off < n) v = v + __shfl_down_sync(0xffffffffu, v, off);
    if (n <= 32) return v;
    if ((lane & 31) == 0) red[lane >> 5] = v;
    sync();
    double r = 0.0;
    if (lane < 32) {
        r = lane < LANES / 32 ? red[lane] : 0.0;
        if (n > 64) r = r + __shfl_down_sync(0xffffffffu, r, 2);
        r = r + __shfl_down_sync(0xffffffffu, r, 1);
    }
    return r;
}

}  // namespace ns3d
