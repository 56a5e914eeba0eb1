// mixed_chunk.cuh -- the FP32 BiCGSTAB loop of small sets without a multilevel
// system: one 1024-row chunk per block, one row per thread (included by
// mixed.cu).
//
// The scheme of krylov_chunk.cuh in FP32.  What bounds a small set is latency:
// k_m32_loop<true> spent 17.6 us on an iteration of 103 chunks, in three grid
// barriers with fences, the reloads after them and the sums of 412 partials.
// Here the block keeps its chunk in shared memory, and y, z and the partials
// travel as single 8-byte words, 32 bits of value and 32 bits of epoch (the
// partials of a work unit are FP32 sums), polled by the readers: no grid
// barrier, no fence, and a neighbour inside the chunk comes from shared
// memory.  The arithmetic and its order are those of k_m32_loop: the row
// products of spmv_f32_row, work units of 256 rows (lane l of a unit
// accumulates rows l and l + 128 in FP32), FP64 sums of the unit partials.
//
// (Two chunks per block for sets of up to twice as many chunks measured slower
// than the other loops: 47 -> 60 ms for two SIMPLER outer iterations at 157
// chunks.)
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
constexpr size_t kMChunkSmemBytes = (size_t)(MCHUNK_ARRAYS + 6) * CH * 4;

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

template <int CAP>
__global__ void __launch_bounds__(CH, 1)
    k_m32_chunk(const __grid_constant__ MSetArgT<CAP> A, GridBar *bar, int max_iters) {
    static_assert(CH == 1024 && MRPL == 2, "one thread per row of a chunk; rows l and l + 128 of a unit");
    static_assert(LOOP_GROUPS == 2 * MSUB, "one group per unit and sum");
    extern __shared__ float sm_m[];
    __shared__ KState st;
    __shared__ double s_sum[2], s_tree[2][8];
    __shared__ float s_ftree[LOOP_GROUPS][4];
    const int t = threadIdx.x, gi = t / LANES, lane = t % LANES;
    const GroupSync sync{gi + 1};
    const MSys &S = A.sys[msys_of_chunk(A, (int)blockIdx.x)];
    const int lc = (int)blockIdx.x - S.chunk_begin, base = lc * CH, row = base + t, units = S.nchunks * MSUB;
    if (t == 0) {
        st = *S.st;
        if (S.dc->done) st.done = 1;
    }
    enum { INVD = 7, R0, X, P, Y, V, SV, Z, T, RV };
    auto arr = [&](int a) { return sm_m + a * CH; };
    int *const col = reinterpret_cast<int *>(arr(MCHUNK_ARRAYS)) + t;
    __syncthreads();
    if (S.dc->done) return;  // the same in every block of the system
    arr(X)[t] = 0.0f;
    {
        const size_t np = (size_t)S.npad;
#pragma unroll
        for (int d = 0; d < 7; ++d) arr(d)[t] = ro(S.coef32 + d * np + row);
#pragma unroll
        for (int d = 0; d < 6; ++d) col[d * CH] = ro(S.nbr + d * np + row);
        arr(INVD)[t] = ro(S.invdiag32 + row);
        const float r = S.r[row];  // k_m32_init: r0 = r, x = p = v = 0
        arr(RV)[t] = r;
        arr(R0)[t] = r;
        arr(P)[t] = 0.0f;
        arr(V)[t] = 0.0f;
    }
    const unsigned int never = bar->bias ? 0x80000000u : 0u;  // as in k_kr_chunk
    int bad = 0;
    auto epoch = [&] { return (unsigned int)st.work + 1u; };
    // row product of the thread's row from its value and its columns'
    auto product = [&](int a, const unsigned long long *words) {
        float xc[6];
        const float *own = arr(a);
        gather_tagged_f32(col, base, t, own, words, epoch(), xc, bar, bad);
        const float *cf = arr(0) + t;
        float acc = cf[0] * own[t];
        acc = __fmaf_rn(cf[1 * CH], xc[0], acc);
        acc = __fmaf_rn(cf[3 * CH], xc[2], acc);
        acc = __fmaf_rn(cf[5 * CH], xc[4], acc);
        acc = __fmaf_rn(cf[6 * CH], xc[5], acc);
        acc = __fmaf_rn(cf[4 * CH], xc[3], acc);
        acc = __fmaf_rn(cf[2 * CH], xc[1], acc);
        return acc;
    };
    // `sums` dot products (kinds kind, kind + 1; operands a_j, b_j) over the
    // system into s_sum: the units' partials by one group each, published,
    // then the sum over the system's units in the fixed order.  false when a
    // wait ran out.
    auto dots = [&](int kind, int sums, int a0, int b0, int a1, int b1) {
        const int sub = gi % MSUB, j = gi / MSUB;
        if (j < sums) {
            const float *a = arr(j ? a1 : a0), *b = arr(j ? b1 : b0);
            float acc = 0.0f;
#pragma unroll
            for (int m = 0; m < MRPL; ++m) {
                const int q = sub * MUNIT + lane + m * LANES;
                if (base + q < S.n) acc = __fmaf_rn(a[q], b[q], acc);
            }
            const float part = lanes_tree_sum<float>(acc, lane, s_ftree[gi], sync);
            if (lane == 0) {
                st_word(unit_tag_words(S) + (size_t)(kind + j) * units + lc * MSUB + sub, tag_f32(part, epoch()));
                // a chunk's four units end together: one of them counts
                if (sub == MSUB - 1) count_arrival(tag_counter(S.part, S.nchunks, kind + j));
            }
        }
        if (gi < sums) {
            const unsigned long long *words = unit_tag_words(S) + (size_t)(kind + gi) * units;
            const unsigned int want = epoch() | never;
            PollLimit limit(bar, bad);
            if (lane == 0)
                wait_arrivals(tag_counter(S.part, S.nchunks, kind + gi), epoch() * (unsigned int)S.nchunks, limit);
            sync();
            double sum = 0.0;
            for (int i = lane; i < units; i += 4 * LANES) {
                unsigned long long w[4];
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (i + m * LANES < units) w[m] = ld_word(words + i + m * LANES);
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (i + m * LANES < units) {
                        while ((unsigned int)(w[m] >> 32) != want && limit.again()) w[m] = ld_word(words + i + m * LANES);
                        sum = sum + (double)__uint_as_float((unsigned int)w[m]);
                    }
            }
            const double v = group_tree(sum, min(units, LANES), lane, s_tree[gi], sync);
            if (lane == 0) s_sum[gi] = v;
        }
        return __syncthreads_or(bad) == 0;
    };
    for (int it = 0; !st.done && it < max_iters; ++it) {
        // p = r + beta (p - w v); y = D^-1 p
        {
            const float beta = (float)st.beta, w = (float)st.w;
            const float p = __fmaf_rn(beta, __fmaf_rn(-w, arr(V)[t], arr(P)[t]), arr(RV)[t]);
            const float y = arr(INVD)[t] * p;
            st_word(S.wy + row, tag_f32(y, epoch()));
            arr(P)[t] = p;
            arr(Y)[t] = y;
        }
        __syncthreads();
        // v = A y, <r0, v>
        arr(V)[t] = product(Y, S.wy);
        if (__syncthreads_or(bad)) break;
        if (!dots(0, 1, R0, V, R0, V)) break;
        if (t == 0) st.alpha = st.rho / s_sum[0];
        __syncthreads();
        // s = r - alpha v; z = D^-1 s
        {
            const float s = __fmaf_rn(-(float)st.alpha, arr(V)[t], arr(RV)[t]);
            const float z = arr(INVD)[t] * s;
            st_word(S.wz + row, tag_f32(z, epoch()));
            arr(SV)[t] = s;
            arr(Z)[t] = z;
        }
        __syncthreads();
        // t = A z, <t, t>, <t, s>
        arr(T)[t] = product(Z, S.wz);
        if (__syncthreads_or(bad)) break;
        if (!dots(1, 2, T, T, T, SV)) break;
        if (t == 0) st.w = (s_sum[0] > 0.0) ? s_sum[1] / s_sum[0] : 0.0;
        __syncthreads();
        // x += alpha y + w z; r = s - w t; <r0, r>, <r, r>
        {
            const float alpha = (float)st.alpha, w = (float)st.w;
            arr(X)[t] = __fmaf_rn(w, arr(Z)[t], __fmaf_rn(alpha, arr(Y)[t], arr(X)[t]));
            arr(RV)[t] = __fmaf_rn(-w, arr(T)[t], arr(SV)[t]);
        }
        __syncthreads();
        if (!dots(3, 2, R0, RV, RV, RV)) break;
        if (t == 0) m32_end_iteration(st, s_sum[0], s_sum[1]);
        __syncthreads();
    }
    // the correction in FP64, for k_dc_step and k_dc_update
    if (st.info == 0) {
        __syncthreads();  // (uniform) s_sum is read
        if (t == 0) s_sum[0] = 1.0 / S.dc->scale;
        __syncthreads();
        S.d64[row] = (double)arr(X)[t] * s_sum[0];
    }
    if (lc == 0 && t == 0) {
        st.counter = 0;
        *S.st = st;
    }
}

}  // namespace ns3d
