// mixed.h -- data of the mixed-precision (FP32 inner / FP64 outer) solves.
#pragma once

#include "device.cuh"

namespace ns3d {

// work unit of the FP32 loop kernel: MRPL rows per lane, MSUB units per chunk
constexpr int MRPL = 2;
constexpr int MUNIT = LANES * MRPL;
constexpr int MSUB = CH / MUNIT;
static_assert(PART_PER_CHUNK >= 5 * MSUB, "partials of the FP32 loop kernel");

// FP64 defect-correction state of one system
struct DCState {
    double rr, bb, tol, tol2, scale, error, tin, tin_min;
    double theta;    // step length of the current correction (minimal FP64 residual)
    int total_iter, maxit, done, info, zero_rhs;
    int inner_cap;   // FP32 iterations allowed per round
    unsigned int counter, pad2_;
};

// Aggregation multilevel preconditioner of an FP32 inner solve (precision
// mode MIXED_MG, single-system sets): level k+1 aggregates the rows of level
// k by 2x2x2 blocks of their cells; its operator is the Galerkin product
// (sum of the block's couplings; blocks couple through faces only, so it is
// 7-point again, same slot order P,W,E,S,N,B,T).
constexpr int MG_MAX = 6;
struct MGLevel {
    int n, npad;
    const int *nbr;       // [6][npad], -1 none
    float *coef;          // [7][npad]
    float *invdiag;       // [npad]
    const int *pos;       // [rows of level k-1]: 8 x the row of this level each belongs to + its rank there
    const int *mstart;    // [n + 1]: offsets into members
    const int *members;   // rows of level k-1 of each row, ascending
    float *x, *b, *t, *xo;  // V-cycle vectors [npad]: Jacobi start, right-hand side, scratch, result
    float *t8;            // [8 npad]: the residual of level k-1 at `pos`, +0 in the unused places
};
struct MGSet {
    int nlev;             // coarse levels (0: Jacobi preconditioning)
    int sweeps;           // Jacobi sweeps on the coarsest level
    float omega;          // damping of the Jacobi smoother
    const ushort4 *pack;  // the system's columns in 8 bytes a row (row_columns) or null
    int tail;             // levels tail..nlev run in every block's shared memory (nlev + 1: none do)
    MGLevel lev[MG_MAX + 1];  // lev[1..nlev]; lev[0] unused (the system itself)
};
// The tail takes the levels from the coarsest up while they have at most this
// many rows together: 85 bytes a row, so the largest tail leaves 90 KB of the
// SM's 256 KB for the L1 that the fine levels' gathers need.
constexpr int MG_TAIL_ROWS = 1792;
// shared memory of the tail (32-bit words), the layout of TailLevels
inline size_t mg_tail_words(const MGSet &mg) {
    size_t w = 0;
    for (int k = mg.tail; k <= mg.nlev; ++k) {
        w += (size_t)18 * mg.lev[k].n;
        if (k > mg.tail) w += (size_t)mg.lev[k].n + 1 + 2 * (size_t)mg.lev[k - 1].n;
    }
    return w;
}

struct MSys {
    int n, npad, nchunks, chunk_begin;
    const int *nbr;
    const double *coef64;  // [7][npad]
    const double *b64;     // right-hand side
    double *x64;           // guess in, solution out
    double *r64;           // FP64 residual
    double *d64;           // the round's correction double(x) / scale, written by the FP32 loop
    const float *coef32, *invdiag32;
    float *x, *r, *r0, *p, *v, *y, *s, *z, *t;  // FP32 inner vectors (x is the correction)
    float *p2, *v2;  // second buffers of p and v (the loop kernel alternates them)
    unsigned long long *wy, *wz;  // words of y and z exchanged by the loop with resident chunks (mixed_chunk.cuh)
    double *part;
    KState *st;  // inner BiCGSTAB state (scalars in FP64)
    DCState *dc;
    MGSet mg;
};

// A mixed solve set as a kernel argument (by value; systems in chunk order):
// one solver instance's systems (up to KMAX) or the systems of many
// concurrent solves (up to KMAX_MERGED_M, 24 KB of kernel parameters).
constexpr int KMAX_MERGED_M = 32;
template <int CAP>
struct MSetArgT {
    int nsys, total_chunks;
    int resident, pad_;  // 1: the loop with resident chunks, 0: the other loops (plan_mixed)
    MSys sys[CAP];
};
using MSetArg = MSetArgT<KMAX>;
using MSetArgMerged = MSetArgT<KMAX_MERGED_M>;
static_assert(sizeof(MSetArgMerged) <= 32000, "kernel parameter space");

// Galerkin operators of every coarse level of `mg` from the FP32 system
void launch_mg_galerkin(const MSys &sys, cudaStream_t st);
void launch_to_f32(const double *coef, const double *invdiag, int npad, float *coef32, float *invdiag32,
                   cudaStream_t st);
// (the set launchers are instantiated for CAP = KMAX and KMAX_MERGED_M)
// chooses the FP32 loop of a solve of the set (kept for all its rounds);
// before the other launches
template <int CAP>
void plan_mixed(MSetArgT<CAP> &set, int share);
template <int CAP>
void launch_dc_resid(const MSetArgT<CAP> &set, int first, cudaStream_t st);
template <int CAP>
void launch_m32_init(const MSetArgT<CAP> &set, cudaStream_t st);
// The FP32 loop variant of a set without resident chunks: fused (three phases
// per iteration) when the set has at most kFusedRows rows and no multilevel
// system, else the five-phase loop.  A merged set runs the variant its members
// chose alone, which is a matter of speed: the bits are the same.
bool m32_fused(long rows, bool mg);
// FP32 inner iterations until every inner solve of the round is done
// (variant: -1 from the set's own rows, 0 five-phase, 1 fused, not asked for
// with resident chunks; a merged set takes 1/share of the SMs)
template <int CAP>
cudaError_t launch_m32_loop(const MSetArgT<CAP> &set, GridBar *bar, int max_iters, cudaStream_t st,
                            int variant = -1, int share = 1);
// theta = <r, A d> / <A d, A d> for the FP32 correction d (FP64 SpMV), then
// x += theta d
template <int CAP>
void launch_dc_update(const MSetArgT<CAP> &set, cudaStream_t st);

}  // namespace ns3d
