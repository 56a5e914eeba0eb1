// CPU restatement of a mixed-precision solve of one system without a
// multilevel hierarchy: FP32 BiCGSTAB rounds inside FP64 defect correction,
// every operation and every sum in the order of the device code (mixed.cu,
// mixed_chunk.cuh).  Built and called by tests/test_gpu_mixed_restatement.py;
// compile without contraction.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

namespace {

constexpr int kLanes = 128, kChunk = 1024, kUnit = 256;

struct System {
    int n;
    const double *coef;  // [7][n]: P, W, E, S, N, B, T
    const int *nbr;      // [6][n]: W, E, S, N, B, T
    std::vector<float> c32, inv32;
};

// halving tree over 128 lane values: inside the warps, then over the warps
template <class T>
T tree(std::vector<T> v) {
    T w[4];
    for (int k = 0; k < 4; ++k) {
        T *u = v.data() + 32 * k;
        for (int off = 16; off >= 1; off >>= 1)
            for (int l = 0; l < off; ++l) u[l] = u[l] + u[l + off];
        w[k] = u[0];
    }
    for (int off = 2; off >= 1; off >>= 1)
        for (int l = 0; l < off; ++l) w[l] = w[l] + w[l + off];
    return w[0];
}

// partials combined by 128 lanes
double combine(const std::vector<double> &part) {
    std::vector<double> lane(kLanes, 0.0);
    for (size_t i = 0; i < part.size(); ++i) lane[i % kLanes] = lane[i % kLanes] + part[i];
    return tree(lane);
}

// sum over blocks of `block` rows: lane l of a block accumulates rows l,
// l + 128, ... with fused multiply-adds in type T, a tree per block, the
// blocks' sums in FP64
template <class T, class Tree>
double dot(const std::vector<T> &a, const std::vector<T> &b, int n, int block, Tree tree_of) {
    std::vector<double> part;
    for (int r0 = 0; r0 < n; r0 += block) {
        std::vector<T> lane(kLanes, T(0));
        for (int r = r0; r < std::min(n, r0 + block); ++r) {
            T &s = lane[(r - r0) % kLanes];
            s = std::fma(a[r], b[r], s);
        }
        part.push_back(tree_of(lane));
    }
    // (a chunk always has all its units; empty ones add zeros)
    const int per_chunk = kChunk / block;
    while (part.size() % per_chunk) part.push_back(0.0);
    return combine(part);
}
double dot64(const std::vector<double> &a, const std::vector<double> &b) {
    return dot(a, b, (int)a.size(), kChunk, [](const std::vector<double> &v) { return tree(v); });
}
double dot32(const std::vector<float> &a, const std::vector<float> &b) {
    return dot(a, b, (int)a.size(), kUnit, [](const std::vector<float> &v) { return (double)tree(v); });
}

// row product in FP64: ascending columns
double row64(const System &S, const std::vector<double> &x, int r) {
    int col[7], slot[7], m = 0;
    for (int d = 0; d < 6; ++d)
        if (S.nbr[(size_t)d * S.n + r] >= 0) {
            col[m] = S.nbr[(size_t)d * S.n + r];
            slot[m++] = d + 1;
        }
    col[m] = r;
    slot[m++] = 0;
    double acc = 0.0;
    for (int k = 0; k < m; ++k) {
        int at = k;
        for (int q = k + 1; q < m; ++q)
            if (col[q] < col[at]) at = q;
        std::swap(col[k], col[at]);
        std::swap(slot[k], slot[at]);
        acc = std::fma(S.coef[(size_t)slot[k] * S.n + r], x[col[k]], acc);
    }
    return acc;
}

// row product in FP32: P, W, S, B, T, N, E; a missing entry is a zero
// coefficient times the row's own value
float row32(const System &S, const std::vector<float> &x, int r) {
    const float *c = S.c32.data() + r;
    const size_t n = S.n;
    auto val = [&](int d) {
        const int k = S.nbr[d * n + r];
        return x[k >= 0 ? k : r];
    };
    float acc = c[0] * x[r];
    for (int d : {0, 2, 4, 5, 3, 1}) acc = std::fma(c[(d + 1) * n], val(d), acc);
    return acc;
}

}  // namespace

extern "C" void mixed_restatement(const double *coef, const int *nbr, const double *b_in, double *x_io, int n, double tol,
                                  int maxit, double inner_tol, int inner_cap, int *iterations, int *info, double *error) {
    System S{n, coef, nbr, std::vector<float>((size_t)7 * n), std::vector<float>(n)};
    for (size_t i = 0; i < (size_t)7 * n; ++i) S.c32[i] = (float)coef[i];
    for (int r = 0; r < n; ++r) S.inv32[r] = (float)(coef[r] != 0.0 ? 1.0 / coef[r] : 1.0);
    std::vector<double> x64(x_io, x_io + n), b(b_in, b_in + n), r64(n), d64(n), q64(n);
    std::vector<float> x(n), r(n), r0(n), p(n), v(n), y(n), s(n), z(n), t(n);
    int total = 0, inner_iter = 0, inner_info = 0;
    double bb = 0, tol2 = 0;
    for (bool first = true;; first = false) {
        for (int i = 0; i < n; ++i) r64[i] = b[i] - row64(S, x64, i);
        const double rr = dot64(r64, r64);
        if (!first) total += inner_iter;
        if (first) {
            bb = dot64(b, b);
            tol2 = tol * tol * bb;
        }
        if (first && bb == 0.0) {
            *iterations = maxit;
            *info = 0;
            *error = tol;
            std::fill(x64.begin(), x64.end(), 0.0);
            break;
        }
        if (!std::isfinite(rr) || (!first && inner_info == 1)) {
            *iterations = total;
            *info = 1;
            *error = std::sqrt(rr / bb);
            break;
        }
        if (!(rr > tol2 && total < maxit)) {
            *iterations = total;
            *error = std::sqrt(rr / bb);
            *info = *error <= tol ? 0 : 2;
            break;
        }
        const double scale = 1.0 / std::sqrt(rr), need = 0.5 * std::sqrt(tol2 / rr);
        const double tin = need > inner_tol ? need : inner_tol;
        const int cap = std::min(inner_cap, maxit - total);
        // FP32 round
        std::vector<double> part;
        for (int i = 0; i < n; ++i) {
            r[i] = r0[i] = (float)(r64[i] * scale);
            x[i] = p[i] = v[i] = 0.0f;
        }
        for (int c0 = 0; c0 < n; c0 += kChunk) {  // |f|^2: FP32 lanes over a chunk, FP64 tree
            std::vector<float> acc(kLanes, 0.0f);
            for (int i = c0; i < std::min(n, c0 + kChunk); ++i) acc[(i - c0) % kLanes] = std::fma(r[i], r[i], acc[(i - c0) % kLanes]);
            part.push_back(tree(std::vector<double>(acc.begin(), acc.end())));
        }
        const double ff = combine(part), in2 = tin * tin * ff;
        double rho = 1.0, alpha = 1.0, w = 1.0, beta = 0.0;
        inner_iter = inner_info = 0;
        bool done = !(ff > in2 && 0 < cap);
        if (!done) beta = rho = ff;
        while (!done) {
            const float fb = (float)beta, fw = (float)w;
            for (int i = 0; i < n; ++i) {
                p[i] = std::fma(fb, std::fma(-fw, v[i], p[i]), r[i]);
                y[i] = S.inv32[i] * p[i];
            }
            for (int i = 0; i < n; ++i) v[i] = row32(S, y, i);
            alpha = rho / dot32(r0, v);
            const float fa = (float)alpha;
            for (int i = 0; i < n; ++i) {
                s[i] = std::fma(-fa, v[i], r[i]);
                z[i] = S.inv32[i] * s[i];
            }
            for (int i = 0; i < n; ++i) t[i] = row32(S, z, i);
            const double tt = dot32(t, t), ts = dot32(t, s);
            w = tt > 0.0 ? ts / tt : 0.0;
            const float fw2 = (float)w;
            for (int i = 0; i < n; ++i) {
                x[i] = std::fma(fw2, z[i], std::fma(fa, y[i], x[i]));
                r[i] = std::fma(-fw2, t[i], s[i]);
            }
            const double f0r = dot32(r0, r), frr = dot32(r, r);
            ++inner_iter;
            if (!std::isfinite(frr) || !std::isfinite(alpha) || !std::isfinite(w)) {
                done = true;
                inner_info = 1;
            } else if (!(frr > in2 && inner_iter < cap)) {
                done = true;
            } else if (std::fabs(f0r) < (double)FLT_EPSILON * FLT_EPSILON * ff || w == 0.0) {
                done = true;
            } else {
                beta = (f0r / rho) * (alpha / w);
                rho = f0r;
            }
        }
        if (inner_info == 0) {
            const double inv = 1.0 / scale;
            for (int i = 0; i < n; ++i) d64[i] = (double)x[i] * inv;
            for (int i = 0; i < n; ++i) q64[i] = row64(S, d64, i);
            const double rq = dot64(r64, q64), qq = dot64(q64, q64);
            double theta = qq > 0.0 ? rq / qq : 0.0;
            if (!std::isfinite(theta)) theta = 0.0;
            for (int i = 0; i < n; ++i) x64[i] = std::fma(theta, d64[i], x64[i]);
        }
    }
    std::copy(x64.begin(), x64.end(), x_io);
}
