// mixed_chunk.cuh -- the FP32 BiCGSTAB loop of small sets without a multilevel
// system: R 1024-row chunks per block, R rows per thread (included by
// mixed.cu).
//
// The scheme of krylov_chunk.cuh in FP32.  What bounds a small set is latency:
// k_m32_loop<true> spent 17.6 us on an iteration of 103 chunks, in three grid
// barriers with fences, the reloads after them and the sums of 412 partials.
// Here the block keeps its chunks in shared memory, and y, z and the partials
// travel as single 8-byte words, 32 bits of value and 32 bits of epoch (the
// partials of a work unit are FP32 sums), polled by the readers: no grid
// barrier, no fence, and a neighbour inside the chunk comes from shared
// memory.  The arithmetic and its order are those of k_m32_loop: the row
// products of spmv_f32_row, work units of 256 rows (lane l of a unit
// accumulates rows l and l + 128 in FP32), FP64 sums of the unit partials.
//
// R = 1 while every chunk gets a block, R = 2 up to twice that (a block's two
// chunks may belong to different systems; every block runs the phases of all
// its chunks in the same order, so no two blocks wait for each other).
//
// The words of y and z live in the FP64 work vectors p and v of the system
// (S.wy, S.wz), those of the partials behind the plain ones in S.part.  They
// are zeroed at the start of a solve (k_dc_zero); the epoch is the system's
// inner iteration count of the solve, starting at 1.  A word is rewritten
// only after every reader has read it, by the argument of krylov_chunk.cuh.
#pragma once

#include "tags.cuh"

namespace ns3d {

// S.part of a system in the FP32 loops: [0, 20 n) plain partials, then one
// word per kind and work unit
__device__ __forceinline__ unsigned long long *unit_tag_words(const MSys &S) {
    return reinterpret_cast<unsigned long long *>(S.part + 5 * MSUB * (size_t)S.nchunks);
}
static_assert(PART_PER_CHUNK >= 5 * MSUB + TAG_KINDS * MSUB, "tagged partials of the work units");

__device__ __forceinline__ unsigned long long tag_f32(float v, unsigned int ep) {
    return ((unsigned long long)ep << 32) | __float_as_uint(v);
}

constexpr int MCHUNK_ARRAYS = 7 + 10;  // coefficients; D^-1, r0, x, p, y, v, s, z, t, r
template <int R>
constexpr size_t kMChunkSmemBytes = (size_t)R * (MCHUNK_ARRAYS + 6) * CH * 4;

// The six column values of a row, slots W, E, S, N, B, T (gather_tagged of
// krylov_chunk.cuh with one word per value; a missing neighbour takes the
// row's own value, its coefficient is zero).
__device__ __forceinline__ void gather_tagged_f32(const int *s_col, int base, int t, const float *own,
                                                  const unsigned long long *words, unsigned int ep, float (&x)[6],
                                                  GridBar *bar, int &bad) {
    unsigned int need = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int c = s_col[d * CH];
        const unsigned int q = (unsigned int)(c - base);
        const bool ext = c >= 0 && q >= (unsigned int)CH;
        x[d] = own[!ext && c >= 0 ? q : t];
        need |= (unsigned int)ext << d;
    }
    PollLimit limit(bar, bad);
    while (need) {
        unsigned long long a[6];
#pragma unroll
        for (int d = 0; d < 6; ++d)
            if (need >> d & 1u) a[d] = ld_word(words + s_col[d * CH]);
#pragma unroll
        for (int d = 0; d < 6; ++d)
            if ((need >> d & 1u) && (unsigned int)(a[d] >> 32) == ep) {
                x[d] = __uint_as_float((unsigned int)a[d]);
                need &= ~(1u << d);
            }
        if (need && !limit.again()) return;
    }
}

template <int CAP, int R>
__global__ void __launch_bounds__(CH, 1)
    k_m32_chunk(const __grid_constant__ MSetArgT<CAP> A, GridBar *bar, int max_iters) {
    static_assert(CH == 1024 && MRPL == 2, "one thread per row of a chunk; rows l and l + 128 of a unit");
    extern __shared__ float sm_m[];
    __shared__ KState sst[R];
    __shared__ double s_sum[R][2], s_tree[R * 2][8];
    __shared__ float s_ftree[8][4];
    const int t = threadIdx.x, gi = t / LANES, lane = t % LANES;
    const GroupSync sync{gi + 1};
    __shared__ int si[R], lc[R];  // system and chunk of slot k (-1: no chunk)
    if (t < R) {
        const int c = (int)blockIdx.x + t * (int)gridDim.x;
        si[t] = c < A.total_chunks ? msys_of_chunk(A, c) : -1;
        lc[t] = si[t] >= 0 ? c - A.sys[si[t]].chunk_begin : 0;
        if (si[t] >= 0) {
            sst[t] = *A.sys[si[t]].st;
            if (A.sys[si[t]].dc->done) sst[t].done = 1;
        }
    }
    enum { INVD = 7, R0, X, P, Y, V, SV, Z, T, RV };
    auto arr = [&](int k, int a) { return sm_m + (k * (MCHUNK_ARRAYS + 6) + a) * CH; };
    auto col = [&](int k) { return reinterpret_cast<int *>(arr(k, MCHUNK_ARRAYS)) + t; };
    __syncthreads();
    auto on = [&](int k) { return si[k] >= 0 && !sst[k].done; };
#pragma unroll
    for (int k = 0; k < R; ++k) {
        arr(k, X)[t] = 0.0f;
        if (!on(k)) continue;
        const MSys &S = A.sys[si[k]];
        const size_t np = (size_t)S.npad;
        const int row = lc[k] * CH + t;
#pragma unroll
        for (int d = 0; d < 7; ++d) arr(k, d)[t] = ro(S.coef32 + d * np + row);
#pragma unroll
        for (int d = 0; d < 6; ++d) col(k)[d * CH] = ro(S.nbr + d * np + row);
        arr(k, INVD)[t] = ro(S.invdiag32 + row);
        const float r = S.r[row];  // k_m32_init: r0 = r, x = p = v = 0
        arr(k, RV)[t] = r;
        arr(k, R0)[t] = r;
        arr(k, P)[t] = 0.0f;
        arr(k, V)[t] = 0.0f;
    }
    const unsigned int never = bar->bias ? 0x80000000u : 0u;  // as in k_kr_chunk
    int bad = 0;
    auto epoch = [&](int k) { return (unsigned int)sst[k].work + 1u; };
    // row product of slot k's row from its value and its columns'
    auto product = [&](int k, int a, const unsigned long long *words) {
        float xc[6];
        const float *own = arr(k, a);
        gather_tagged_f32(col(k), lc[k] * CH, t, own, words, epoch(k), xc, bar, bad);
        const float *cf = arr(k, 0) + t;
        float acc = cf[0] * own[t];
        acc = __fmaf_rn(cf[1 * CH], xc[0], acc);
        acc = __fmaf_rn(cf[3 * CH], xc[2], acc);
        acc = __fmaf_rn(cf[5 * CH], xc[4], acc);
        acc = __fmaf_rn(cf[6 * CH], xc[5], acc);
        acc = __fmaf_rn(cf[4 * CH], xc[3], acc);
        acc = __fmaf_rn(cf[2 * CH], xc[1], acc);
        return acc;
    };
    // `sums` dot products (kinds kind, kind + 1; operands a_j, b_j) of every
    // active slot's system into s_sum: the units' partials by one group each,
    // published, then the sum over the system's units in the fixed order.
    // false when a wait ran out.
    auto dots = [&](int kind, int sums, int a0, int b0, int a1, int b1) {
#pragma unroll 1
        for (int task = gi; task < R * MSUB * sums; task += LOOP_GROUPS) {
            const int unit = task % (R * MSUB), j = task / (R * MSUB), k = unit / MSUB, sub = unit % MSUB;
            if (!on(k)) continue;
            const MSys &S = A.sys[si[k]];
            const float *a = arr(k, j ? a1 : a0), *b = arr(k, j ? b1 : b0);
            const int rows = S.n - lc[k] * CH;
            float acc = 0.0f;
#pragma unroll
            for (int m = 0; m < MRPL; ++m) {
                const int q = sub * MUNIT + lane + m * LANES;
                if (q < rows) acc = __fmaf_rn(a[q], b[q], acc);
            }
            const float part = lanes_tree_sum<float>(acc, lane, s_ftree[gi], sync);
            if (lane == 0) {
                const int n = S.nchunks * MSUB;
                st_word(unit_tag_words(S) + (size_t)(kind + j) * n + lc[k] * MSUB + sub, tag_f32(part, epoch(k)));
                // a chunk's four units end together: one of them counts
                if (sub == MSUB - 1) count_arrival(tag_counter(S.part, S.nchunks, kind + j));
            }
        }
        if (gi < R * sums) {
            const int k = gi / sums, j = gi % sums;
            if (on(k)) {
                const MSys &S = A.sys[si[k]];
                const int n = S.nchunks * MSUB;
                const unsigned long long *words = unit_tag_words(S) + (size_t)(kind + j) * n;
                const unsigned int want = epoch(k) | never;
                PollLimit limit(bar, bad);
                if (lane == 0)
                    wait_arrivals(tag_counter(S.part, S.nchunks, kind + j), epoch(k) * (unsigned int)S.nchunks, limit);
                sync();
                double sum = 0.0;
                for (int base = lane; base < n; base += 4 * LANES) {
                    unsigned long long w[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (base + m * LANES < n) w[m] = ld_word(words + base + m * LANES);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (base + m * LANES < n) {
                            while ((unsigned int)(w[m] >> 32) != want && limit.again())
                                w[m] = ld_word(words + base + m * LANES);
                            sum = sum + (double)__uint_as_float((unsigned int)w[m]);
                        }
                }
                const double v = group_tree(sum, min(n, LANES), lane, s_tree[gi], sync);
                if (lane == 0) s_sum[k][j] = v;
            }
        }
        return __syncthreads_or(bad) == 0;
    };
    bool any = false;
#pragma unroll
    for (int k = 0; k < R; ++k) any = any || on(k);
    for (int it = 0; any && it < max_iters; ++it) {
        // p = r + beta (p - w v); y = D^-1 p
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (!on(k)) continue;
            const float beta = (float)sst[k].beta, w = (float)sst[k].w;
            const float p = __fmaf_rn(beta, __fmaf_rn(-w, arr(k, V)[t], arr(k, P)[t]), arr(k, RV)[t]);
            const float y = arr(k, INVD)[t] * p;
            st_word(A.sys[si[k]].wy + lc[k] * CH + t, tag_f32(y, epoch(k)));
            arr(k, P)[t] = p;
            arr(k, Y)[t] = y;
        }
        __syncthreads();
        // v = A y, <r0, v>
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on(k)) arr(k, V)[t] = product(k, Y, A.sys[si[k]].wy);
        if (__syncthreads_or(bad)) break;
        if (!dots(0, 1, R0, V, R0, V)) break;
        if (t < R && on(t)) sst[t].alpha = sst[t].rho / s_sum[t][0];
        __syncthreads();
        // s = r - alpha v; z = D^-1 s
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (!on(k)) continue;
            const float s = __fmaf_rn(-(float)sst[k].alpha, arr(k, V)[t], arr(k, RV)[t]);
            const float z = arr(k, INVD)[t] * s;
            st_word(A.sys[si[k]].wz + lc[k] * CH + t, tag_f32(z, epoch(k)));
            arr(k, SV)[t] = s;
            arr(k, Z)[t] = z;
        }
        __syncthreads();
        // t = A z, <t, t>, <t, s>
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (on(k)) arr(k, T)[t] = product(k, Z, A.sys[si[k]].wz);
        if (__syncthreads_or(bad)) break;
        if (!dots(1, 2, T, T, T, SV)) break;
        if (t < R && on(t)) sst[t].w = (s_sum[t][0] > 0.0) ? s_sum[t][1] / s_sum[t][0] : 0.0;
        __syncthreads();
        // x += alpha y + w z; r = s - w t; <r0, r>, <r, r>
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (!on(k)) continue;
            const float alpha = (float)sst[k].alpha, w = (float)sst[k].w;
            arr(k, X)[t] = __fmaf_rn(w, arr(k, Z)[t], __fmaf_rn(alpha, arr(k, Y)[t], arr(k, X)[t]));
            arr(k, RV)[t] = __fmaf_rn(-w, arr(k, T)[t], arr(k, SV)[t]);
        }
        __syncthreads();
        if (!dots(3, 2, R0, RV, RV, RV)) break;
        if (t < R && on(t)) m32_end_iteration(sst[t], s_sum[t][0], s_sum[t][1]);
        __syncthreads();
        any = false;
#pragma unroll
        for (int k = 0; k < R; ++k) any = any || on(k);
    }
    // the correction in FP64, for k_dc_step and k_dc_update
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (si[k] < 0) continue;
        const MSys &S = A.sys[si[k]];
        if (S.dc->done || sst[k].info != 0) continue;
        if (t == 0) s_sum[k][0] = 1.0 / S.dc->scale;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (si[k] < 0) continue;
        const MSys &S = A.sys[si[k]];
        if (!(S.dc->done || sst[k].info != 0)) S.d64[lc[k] * CH + t] = (double)arr(k, X)[t] * s_sum[k][0];
        if (lc[k] == 0 && t == 0 && !S.dc->done) {
            sst[k].counter = 0;
            *S.st = sst[k];
        }
    }
}

}  // namespace ns3d
