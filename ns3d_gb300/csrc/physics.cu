// physics.cu -- assembly, corrections and diagnostics of the NS3D solve.
//
// One thread per row of the system being built (rows are the compacted
// nodes, row -> cell through the `cell` table), so every coefficient is
// written once and coalesced.  The arithmetic of each row follows the
// reference expression by expression (cited per kernel); this file is
// compiled with --fmad=false so nothing is contracted.
#include "device.cuh"
#include "kernels.h"

namespace ns3d {

__device__ __forceinline__ double min0(double F) { return (0.0 < F) ? 0.0 : F; }
__device__ __forceinline__ double max0(double F) { return (F < 0.0) ? 0.0 : F; }

__device__ __forceinline__ void finish_momentum_row(const SysView &A, int r, double D, double aW, double aE, double aS,
                                                    double aN, double aB, double aT) {
    A.c(SP, r) = D;
    A.c(SW, r) = aW;
    A.c(SE, r) = aE;
    A.c(SS, r) = aS;
    A.c(SN, r) = aN;
    A.c(SB, r) = aB;
    A.c(ST, r) = aT;
    const int nW = A.nb(0, r), nE = A.nb(1, r), nS = A.nb(2, r), nN = A.nb(3, r), nB = A.nb(4, r), nT = A.nb(5, r);
    double cf[7] = {D, aW, aE, aS, aN, aB, aT};
    // uA.row(r).sum(): stored entries in ascending column order, plain adds
    A.rowsum[r] = row_ordered(r, nW, nE, nS, nN, nB, nT, [&](double acc, int s, int) { return acc + cf[s]; });
    // DiagonalPreconditioner: 1/a_rr, or 1 for a zero diagonal
    A.invdiag[r] = (D != 0.0) ? 1.0 / D : 1.0;
}

// One face of a momentum row between two nodes of the component's own grid:
// D -= ..., a = ... as the reference's upwind (Peclet-like number above
// 2 mu schemefactor) or central form.
//
// PLAIN is the form for schemefactor == 0 and ordinary magnitudes
// (plain_momentum): the same bits from half the FP64 operations, which are
// what bounds the assembly (2 per clock and SM).  With schemefactor == 0 a
// cross face is upwind unless its flux is zero, and then the two forms agree;
// halving is exact, so 0.5 goes into rho; -c - h = -(c + h), and c + 0 = c, so
// each side needs one sum; signs are read from the high words.  What is
// excluded by plain_momentum's ranges: products that underflow where c would
// not absorb them.  Whole solves: six SIMPLEC outer iterations at 159^3 (3.5 M
// rows a component) 205.5 -> 200.1 ms, forty at 64^3 88.7 -> 86.8 ms.

// Cross face: s = sum of the two velocities of the face, F = PLUS ? vm rho id
// : -vm rho id with vm = s/2; c = mu id^2.
template <bool PLAIN, bool PLUS, bool RHO_FIRST>
__device__ __forceinline__ void cross_face(double s, const Phys &ph, double d, double id, double c, double &D,
                                           double &a) {
    if (PLAIN) {
        const double h = (s * (0.5 * ph.rho)) * id;  // |F|, sign of vm
        const double t = c + fabs(h);
        const long long bits = __double_as_longlong(h);
        const bool nan = (unsigned long long)(bits << 1) > 0xffe0000000000000ull;
        const bool into = PLUS ? bits < 0 : bits >= 0;  // F < 0 (or F = 0: t = c)
        D -= (into || nan) ? t : c;
        a = (into && !nan) ? c : t;
    } else {
        const double vm = s * 0.5;
        const double F = PLUS ? vm * ph.rho * id : -vm * ph.rho * id;
        const double pe = RHO_FIRST ? fabs(vm) * ph.rho * d : fabs(vm) * d * ph.rho;
        if (pe > 2 * ph.mu * ph.schemefactor) {
            D += -c + min0(F);
            a = c + max0(F);
        } else {
            D += -c + F * 0.5;
            a = c + F * 0.5;
        }
    }
}

// Face to a neighbour along the component: own velocity o, the neighbour's e;
// the flux is taken from the upstream node if both have one sign.
template <bool PLAIN, bool PLUS>
__device__ __forceinline__ void own_face(double o, double e, const Phys &ph, double d, double id, double c, double &D,
                                         double &a) {
    if (PLAIN) {
        const int ho = __double2hiint(o), he = __double2hiint(e);
        const unsigned int mo = ho & 0x7fffffff, me = he & 0x7fffffff;
        // both of a magnitude within 2^-664..2^664: no sign test meets a zero
        // or NaN, and no flux under- or overflows
        if (min(mo, me) >= 0x16700000u && max(mo, me) < 0x69700000u) {
            const bool same = (ho ^ he) >= 0, up = PLUS ? ho < 0 : ho >= 0;  // up: own node is upstream
            const double x = same ? (up ? o : e) : o + e;
            const double h = (x * (same ? ph.rho : 0.25 * ph.rho)) * id;
            const double lo = c - h, hi = c + h;  // F = h (PLUS) or -h
            D -= (same && !up) ? c : (PLUS ? lo : hi);
            a = (same && up) ? c : (PLUS ? hi : lo);
            return;
        }
    }
    double F;
    if (PLUS ? (o < 0 && e < 0) : (o > 0 && e > 0)) F = PLUS ? o * ph.rho * id : -o * ph.rho * id;
    else if (PLUS ? (o > 0 && e > 0) : (o < 0 && e < 0)) F = PLUS ? e * ph.rho * id : -e * ph.rho * id;
    else F = 0;
    if (fabs(F) * d * d > 2 * ph.mu * ph.schemefactor) {
        D += -c + min0(F);
        a = c + max0(F);
    } else {
        const double m = (o + e) * 0.5;
        const double Fd = PLUS ? m * ph.rho * id : -m * ph.rho * id;
        D += -c + Fd * 0.5;
        a = c + Fd * 0.5;
    }
}

// AssembleMomentum_x, src/NSBase.cxx:886-1057
template <bool PLAIN>
__global__ void k_mom_x(Grid g, Phys ph, SysView A, const double *__restrict__ uc, const double *__restrict__ vc,
                        const double *__restrict__ wc) {
    const double dx = ph.dx, dy = ph.dy, dz = ph.dz, rho = ph.rho;
    const double cx = ph.mu * ph.idx2, cy = ph.mu * ph.idy2, cz = ph.mu * ph.idz2;
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    const int d0 = g.nx + 1, ny = g.ny, nz = g.nz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(A.cell[r], i, j, k);
        double D = 0;
        double aW = 0, aE = 0, aS = 0, aN = 0, aB = 0, aT = 0;
        const double uC = uc[r];
        const int nE = A.nb(1, r), nW = A.nb(0, r);
        if (i + 1 < d0) {
            if (nE > -1) {
                own_face<PLAIN, false>(uC, uc[nE], ph, dx, idx, cx, D, aE);
            } else {
                D += -cx - (0.25 * rho * idx) * (uC);
            }
        } else {
            D += -(rho * idx) * (uC);
        }
        if (i - 1 >= 0) {
            if (nW > -1) {
                own_face<PLAIN, true>(uC, uc[nW], ph, dx, idx, cx, D, aW);
            } else {
                D += -cx + (0.25 * rho * idx) * (uC);
            }
        } else {
            D += (rho * idx) * (uC);
        }
        if (j + 1 < ny) {
            if (A.nb(3, r) > -1) {
                cross_face<PLAIN, false, true>(g.sv(vc, i - 1, j + 1, k) + g.sv(vc, i, j + 1, k),
                                               ph, dy, idy, cy, D, aN);
            } else {
                D += -2 * ph.mu * ph.idy2;
            }
        } else {
            D += -2 * ph.mu * ph.idy2;
        }
        if (j - 1 >= 0) {
            if (A.nb(2, r) > -1) {
                cross_face<PLAIN, true, false>(g.sv(vc, i - 1, j, k) + g.sv(vc, i, j, k), ph, dy, idy, cy, D, aS);
            } else {
                D += -2 * ph.mu * ph.idy2;
            }
        } else {
            D += -2 * ph.mu * ph.idy2;
        }
        if (nz > 1) {
            if (k + 1 < nz) {
                if (A.nb(5, r) > -1) {
                    cross_face<PLAIN, false, true>(g.sw(wc, i - 1, j, k + 1) + g.sw(wc, i, j, k + 1),
                                                   ph, dz, idz, cz, D, aT);
                } else {
                    D += -2 * ph.mu * ph.idz2;
                }
            } else {
                D += -2 * ph.mu * ph.idz2;
            }
            if (k - 1 >= 0) {
                if (A.nb(4, r) > -1) {
                    cross_face<PLAIN, true, true>(g.sw(wc, i - 1, j, k) + g.sw(wc, i, j, k), ph, dz, idz, cz, D, aB);
                } else {
                    D += -2 * ph.mu * ph.idz2;
                }
            } else {
                D += -2 * ph.mu * ph.idz2;
            }
        }
        if (ph.alpha != 1) D /= ph.alpha;
        finish_momentum_row(A, r, D, aW, aE, aS, aN, aB, aT);
    }
}

// AssembleMomentum_y, src/NSBase.cxx:1059-1250
template <bool PLAIN>
__global__ void k_mom_y(Grid g, Phys ph, SysView A, const double *__restrict__ uc, const double *__restrict__ vc,
                        const double *__restrict__ wc) {
    const double dx = ph.dx, dy = ph.dy, dz = ph.dz, rho = ph.rho;
    const double cx = ph.mu * ph.idx2, cy = ph.mu * ph.idy2, cz = ph.mu * ph.idz2;
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    const int d0 = g.nx, ny = g.ny, nz = g.nz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(A.cell[r], i, j, k);
        double D = 0;
        double aW = 0, aE = 0, aS = 0, aN = 0, aB = 0, aT = 0;
        if (i + 1 < d0) {
            if (A.nb(1, r) > -1) {
                cross_face<PLAIN, false, false>(g.su(uc, i + 1, j - 1, k) + g.su(uc, i + 1, j, k),
                                                ph, dx, idx, cx, D, aE);
            } else {
                D += -2 * ph.mu * ph.idx2;
            }
        } else {
            D += -(0.5 * rho * idx) * (g.su(uc, i + 1, j - 1, k) + g.su(uc, i + 1, j, k));
        }
        if (i - 1 >= 0) {
            if (A.nb(0, r) > -1) {
                cross_face<PLAIN, true, false>(g.su(uc, i, j - 1, k) + g.su(uc, i, j, k), ph, dx, idx, cx, D, aW);
            } else {
                D += -2 * ph.mu * ph.idx2;
            }
        } else {
            D += -cx + (0.25 * rho * idx) * (g.su(uc, i, j - 1, k) + g.su(uc, i, j, k));
        }
        const double vC = vc[r];
        const int nN = A.nb(3, r), nS = A.nb(2, r);
        if (j + 1 < ny) {
            if (nN > -1) {
                own_face<PLAIN, false>(vC, vc[nN], ph, dy, idy, cy, D, aN);
            } else {
                D += -cy - (0.25 * rho * idy) * (vC);
            }
        } else {
            D += -cy - (0.25 * rho * idy) * (vC);
        }
        if (j - 1 >= 0) {
            if (nS > -1) {
                own_face<PLAIN, true>(vC, vc[nS], ph, dy, idy, cy, D, aS);
            } else {
                D += -cy + (0.25 * rho * idy) * (vC);
            }
        } else {
            D += -cy + (0.25 * rho * idy) * (vC);
        }
        if (nz > 1) {
            if (k + 1 < nz) {
                if (A.nb(5, r) > -1) {
                    cross_face<PLAIN, false, true>(g.sw(wc, i, j - 1, k + 1) + g.sw(wc, i, j, k + 1),
                                                   ph, dz, idz, cz, D, aT);
                } else {
                    D += -2 * ph.mu * ph.idz2;
                }
            } else {
                D += -2 * ph.mu * ph.idz2;
            }
            if (k - 1 >= 0) {
                if (A.nb(4, r) > -1) {
                    cross_face<PLAIN, true, true>(g.sw(wc, i, j - 1, k) + g.sw(wc, i, j, k), ph, dz, idz, cz, D, aB);
                } else {
                    D += -2 * ph.mu * ph.idz2;
                }
            } else {
                D += -2 * ph.mu * ph.idz2;
            }
        }
        if (ph.alpha != 1) D /= ph.alpha;
        finish_momentum_row(A, r, D, aW, aE, aS, aN, aB, aT);
    }
}

// AssembleMomentum_z, src/NSBase.cxx:1252-1442
template <bool PLAIN>
__global__ void k_mom_z(Grid g, Phys ph, SysView A, const double *__restrict__ uc, const double *__restrict__ vc,
                        const double *__restrict__ wc) {
    const double dx = ph.dx, dy = ph.dy, dz = ph.dz, rho = ph.rho;
    const double cx = ph.mu * ph.idx2, cy = ph.mu * ph.idy2, cz = ph.mu * ph.idz2;
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    const int d0 = g.nx, ny = g.ny, nz = g.nz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(A.cell[r], i, j, k);
        double D = 0;
        double aW = 0, aE = 0, aS = 0, aN = 0, aB = 0, aT = 0;
        if (i + 1 < d0) {
            if (A.nb(1, r) > -1) {
                cross_face<PLAIN, false, false>(g.su(uc, i + 1, j, k - 1) + g.su(uc, i + 1, j, k),
                                                ph, dx, idx, cx, D, aE);
            } else {
                D += -2 * ph.mu * ph.idx2;
            }
        } else {
            D += -(0.5 * rho * idx) * (g.su(uc, i + 1, j, k - 1) + g.su(uc, i + 1, j, k));
        }
        if (i - 1 >= 0) {
            if (A.nb(0, r) > -1) {
                cross_face<PLAIN, true, false>(g.su(uc, i, j, k - 1) + g.su(uc, i, j, k), ph, dx, idx, cx, D, aW);
            } else {
                D += -2 * ph.mu * ph.idx2;
            }
        } else {
            D += -cx + (0.25 * rho * idx) * (g.su(uc, i, j, k - 1) + g.su(uc, i, j, k));
        }
        if (j + 1 < ny) {
            if (A.nb(3, r) > -1) {
                cross_face<PLAIN, false, true>(g.sv(vc, i, j + 1, k - 1) + g.sv(vc, i, j + 1, k),
                                               ph, dy, idy, cy, D, aN);
            } else {
                D += -2 * ph.mu * ph.idy2;
            }
        } else {
            D += -2 * ph.mu * ph.idy2;
        }
        if (j - 1 >= 0) {
            if (A.nb(2, r) > -1) {
                cross_face<PLAIN, true, true>(g.sv(vc, i, j, k - 1) + g.sv(vc, i, j, k), ph, dy, idy, cy, D, aS);
            } else {
                D += -2 * ph.mu * ph.idy2;
            }
        } else {
            D += -2 * ph.mu * ph.idy2;
        }
        const double wC = wc[r];
        const int nT = A.nb(5, r), nB = A.nb(4, r);
        if (k + 1 < nz) {
            if (nT > -1) {
                own_face<PLAIN, false>(wC, wc[nT], ph, dz, idz, cz, D, aT);
            } else {
                D += -cz - (0.25 * rho * idz) * (wC);
            }
        } else {
            D += -cz - (0.25 * rho * idz) * (wC);
        }
        if (k - 1 >= 0) {
            if (nB > -1) {
                own_face<PLAIN, true>(wC, wc[nB], ph, dz, idz, cz, D, aB);
            } else {
                D += -cz + (0.25 * rho * idz) * (wC);
            }
        } else {
            D += -cz + (0.25 * rho * idz) * (wC);
        }
        if (ph.alpha != 1) D /= ph.alpha;
        finish_momentum_row(A, r, D, aW, aE, aS, aN, aB, aT);
    }
}

// Assemble_RHS_u/v/w, src/NSBase.cxx:1445-1546
template <int COMP>
__global__ void k_mom_rhs(Grid g, Phys ph, SysView A, const double *__restrict__ p, const double *__restrict__ x) {
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(A.cell[r], i, j, k);
        double b;
        if (COMP == 0) {
            if (i == 0) b = (p[g.P(i, j, k)] - ph.p0) * idx;
            else if (i == g.nx) b = (ph.p1 - p[g.P(i - 1, j, k)]) * idx;
            else b = (p[g.P(i, j, k)] - p[g.P(i - 1, j, k)]) * idx;
            b += x[r] * A.c(SP, r) * (1 - ph.alpha);
        } else if (COMP == 1) {
            b = (p[g.P(i, j, k)] - p[g.P(i, j - 1, k)]) * idy + x[r] * A.c(SP, r) * (1 - ph.alpha);
        } else {
            b = (p[g.P(i, j, k)] - p[g.P(i, j, k - 1)]) * idz + x[r] * A.c(SP, r) * (1 - ph.alpha);
        }
        A.rhs[r] = b;
    }
}

// Compute_{u,v,w}_hat, src/NSBase.cxx:1548-1755: subtractions in the order
// E, W, N, S, T, B, then division by the (relaxed) diagonal
__global__ void k_hat(SysView A, Phys ph, const double *__restrict__ xc, const double *__restrict__ xold,
                      double *__restrict__ hat) {
    const int order[6] = {SE, SW, SN, SS, ST, SB};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        double t = 0;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            int s = order[q];
            int c = A.nb(s - 1, r);
            if (c >= 0) t -= A.c(s, r) * xc[c];
        }
        hat[r] = (t) / (A.c(SP, r)) + xold[r] * (1 - ph.alpha);
    }
}

// AssemblePressure (mode 0, src/NSBase.cxx:478-610),
// AssemblePressureCorrectionSIMPLEC (mode 1, :612-732), ...SIMPLE (mode 2, :734-851)
__global__ void k_pressure(int mode, int relax, Grid g, Phys ph, SysView S, const double *__restrict__ au,
                           const double *__restrict__ av, const double *__restrict__ aw, const double *__restrict__ uc,
                           const double *__restrict__ vc, const double *__restrict__ wc, const double *__restrict__ p) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const double dx2 = ph.dx * ph.dx, dy2 = ph.dy * ph.dy, dz2 = ph.dz * ph.dz;
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(S.cell[r], i, j, k);
        double D = 0, b = 0;
        double cW = 0, cE = 0, cS = 0, cN = 0, cB = 0, cT = 0;
        int f;
        if (i > 0 && g.P(i - 1, j, k) > -1 && (f = g.U(i, j, k)) > -1) {
            D += 1 / ((au[f]) * dx2);
            cW = -1 / ((au[f]) * dx2);
            b -= uc[f] * idx;
        }
        if (i < nx - 1 && g.P(i + 1, j, k) > -1 && (f = g.U(i + 1, j, k)) > -1) {
            D += 1 / ((au[f]) * dx2);
            cE = -1 / ((au[f]) * dx2);
            b += uc[f] * idx;
        }
        if (j > 0 && g.P(i, j - 1, k) > -1 && (f = g.V(i, j, k)) > -1) {
            D += 1 / ((av[f]) * dy2);
            cS = -1 / ((av[f]) * dy2);
            b -= vc[f] * idy;
        }
        if (j < ny - 1 && g.P(i, j + 1, k) > -1 && (f = g.V(i, j + 1, k)) > -1) {
            D += 1 / ((av[f]) * dy2);
            cN = -1 / ((av[f]) * dy2);
            b += vc[f] * idy;
        }
        if (k > 0 && g.P(i, j, k - 1) > -1 && (f = g.W(i, j, k)) > -1) {
            D += 1 / ((aw[f]) * dz2);
            cB = -1 / ((aw[f]) * dz2);
            b -= wc[f] * idz;
        }
        if (k < nz - 1 && g.P(i, j, k + 1) > -1 && (f = g.W(i, j, k + 1)) > -1) {
            D += 1 / ((aw[f]) * dz2);
            cT = -1 / ((aw[f]) * dz2);
            b += wc[f] * idz;
        }
        if (i == 0 && (f = g.U(i, j, k)) > -1) {
            D += 1 / ((au[f]) * dx2);
            if (mode == 0) b -= uc[f] * idx - ph.p0 / (au[f] * dx2);
            else b -= uc[f] * idx;
        }
        if (i == nx - 1 && (f = g.U(i + 1, j, k)) > -1) {
            D += 1 / ((au[f]) * dx2);
            if (mode == 0) b += uc[f] * idx + ph.p1 / (au[f] * dx2);
            else b += uc[f] * idx;
        }
        if (mode == 0 && relax) {
            D /= ph.beta;
            b += p[r] * D * (1 - ph.beta);
        }
        S.c(SP, r) = D;
        S.c(SW, r) = cW;
        S.c(SE, r) = cE;
        S.c(SS, r) = cS;
        S.c(SN, r) = cN;
        S.c(SB, r) = cB;
        S.c(ST, r) = cT;
        S.rhs[r] = b;
        S.invdiag[r] = (D != 0.0) ? 1.0 / D : 1.0;
    }
}

__device__ __forceinline__ double clampdv(double d, double m) {
    if (d < 0 && fabs(d) > m) d = -m;
    else if (d > 0 && d > m) d = m;
    return d;
}

// CorrectVelocityFieldSIMPLE / ...SIMPLEC (src/NSBase.cxx:2082-2263), one
// thread per face node: each face is corrected by exactly one pressure cell
// (its +side cell, or cell nx-1 for the outlet faces), as in the reference
template <int COMP>
__global__ void k_correct(Grid g, Phys ph, SysView A, const double *__restrict__ den, const double *__restrict__ pc,
                          double *__restrict__ x, double dvmax) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k, q, c;
        g.ijk(A.cell[r], i, j, k);
        double d;
        if (COMP == 0) {
            if (i == g.nx) {  // outlet face, owned by cell nx-1
                c = g.P(i - 1, j, k);
                if (c < 0) continue;
                d = -(pc[c]) / ((den[r]) * ph.dx);
            } else if (i == 0) {  // inlet face
                c = g.P(i, j, k);
                if (c < 0) continue;
                d = (pc[c]) / ((den[r]) * ph.dx);
            } else {
                c = g.P(i, j, k);
                q = g.P(i - 1, j, k);
                if (c < 0 || q < 0) continue;
                d = -(pc[q] - pc[c]) / ((den[r]) * ph.dx);
            }
        } else if (COMP == 1) {
            c = g.P(i, j, k);
            q = (j > 0) ? g.P(i, j - 1, k) : -1;
            if (c < 0 || q < 0) continue;
            d = -(pc[q] - pc[c]) / ((den[r]) * ph.dy);
        } else {
            c = g.P(i, j, k);
            q = (k > 0) ? g.P(i, j, k - 1) : -1;
            if (c < 0 || q < 0) continue;
            d = -(pc[q] - pc[c]) / ((den[r]) * ph.dz);
        }
        x[r] = x[r] + clampdv(d, dvmax);
    }
}

// CorrectVelocityFieldSIMPLER, src/NSBase.cxx:2265-2335 (face-parallel)
template <int COMP>
__global__ void k_correct_simpler(Grid g, Phys ph, SysView A, const double *__restrict__ p,
                                  const double *__restrict__ hat, double *__restrict__ x, double p_0, double p_1) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
        int i, j, k, q, c;
        g.ijk(A.cell[r], i, j, k);
        const double a = A.c(SP, r);
        if (COMP == 0) {
            if (i == g.nx) {
                c = g.P(i - 1, j, k);
                if (c < 0) continue;
                x[r] = hat[r] - (p[c] - p_1) / (a * ph.dx);
            } else if (i == 0) {
                c = g.P(i, j, k);
                if (c < 0) continue;
                x[r] = hat[r] - (p_0 - p[c]) / (a * ph.dx);
            } else {
                c = g.P(i, j, k);
                q = g.P(i - 1, j, k);
                if (c < 0 || q < 0) continue;
                x[r] = hat[r] - (p[q] - p[c]) / (a * ph.dx);
            }
        } else if (COMP == 1) {
            c = g.P(i, j, k);
            q = (j > 0) ? g.P(i, j - 1, k) : -1;
            if (c < 0 || q < 0) continue;
            x[r] = hat[r] - (p[q] - p[c]) / (a * ph.dy);
        } else {
            c = g.P(i, j, k);
            q = (k > 0) ? g.P(i, j, k - 1) : -1;
            if (c < 0 || q < 0) continue;
            x[r] = hat[r] - (p[q] - p[c]) / (a * ph.dz);
        }
    }
}

// ComputeVelocityField tail, src/NSBase.cxx:1800-1818: keep the previous
// field when the solve took 0 iterations or failed, then clamp the update
__global__ void k_velocity_post(const double *__restrict__ temp, double *__restrict__ x, int n,
                                const KState *__restrict__ st, int limit, double dvmax) {
    const bool revert = (st->iter == 0) || (st->info != 0);
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        double t = temp[r];
        double v = revert ? t : x[r];
        if (limit) {
            double d = v - t;
            if (fabs(d) > dvmax) {
                if (d > 0) v = t + dvmax;
                else if (d < 0) v = t - dvmax;
            }
        }
        x[r] = v;
    }
}

// ---- reductions with last-block completion ---------------------------------
// Each block reduces whole 1024-row chunks; the block that completes the last
// chunk combines the chunk partials in fixed order and publishes the result.
__device__ __forceinline__ bool last_block_arrive(unsigned int *counter, unsigned int total, bool *sh_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int prev = atomicAdd(counter, 1u);
        *sh_flag = (prev == total - 1);
    }
    __syncthreads();
    bool last = *sh_flag;
    if (last) __threadfence();
    return last;
}

// ComputePermeability, src/NSBase.cxx:1886-1956: sums over the outlet u plane
// (and, with a border, the inlet/outlet p planes), positions q = j*nz + k.
// One plane position per thread, a position without a node adds +0 (which
// changes no sum that starts at +0); group g accumulates sum g.
__global__ void __launch_bounds__(CH) k_permeability(Grid g, const double *__restrict__ u, const double *__restrict__ p,
                                                     int border, double *__restrict__ part, DiagOut *out) {
    __shared__ double s_v[3][CH], sm[12];
    __shared__ bool last;
    const long plane = (long)g.ny * g.nz;
    const int nch = (int)((plane + CH - 1) / CH);
    const int iu = (border <= 0) ? g.nx : g.nx + 1 - border;
    const int io = g.nx - border, ii = border - 1;
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES, sums = border > 0 ? 3 : 1;
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const long q = (long)c * CH + threadIdx.x;
        int ro = -1, ri = -1;
        if (q < plane) {
            const int r = g.umap[(long)iu * plane + q];
            if (border > 0) {
                ro = g.pmap[(long)io * plane + q];
                ri = g.pmap[(long)ii * plane + q];
            }
            s_v[0][threadIdx.x] = r > -1 ? u[r] : 0.0;
            s_v[1][threadIdx.x] = ro > -1 ? p[ro] : 0.0;
            s_v[2][threadIdx.x] = ri > -1 ? p[ri] : 0.0;
        }
        const int co = __syncthreads_count(ro > -1), ci = __syncthreads_count(ri > -1);
        if (gi < sums) {
            const int rows = (int)min((long)CH, plane - (long)c * CH);
            double a = 0.0;
#pragma unroll
            for (int m = 0; m < RPL; ++m)
                if (lane + m * LANES < rows) a = a + s_v[gi][lane + m * LANES];
            const double t = lanes_tree_sum<double>(a, lane, sm + 4 * gi, GroupSync{gi + 1});
            if (lane == 0) part[(size_t)c * 5 + gi] = t;
        }
        if (threadIdx.x == 0) {
            part[(size_t)c * 5 + 3] = (double)co;
            part[(size_t)c * 5 + 4] = (double)ci;
        }
        if (last_block_arrive(&out->counter[0], (unsigned)nch, &last) && gi < 3) {
            const GroupSync sync{gi + 1};
            const double t = gi < sums ? lanes_final_sum(part + gi, nch, 5, lane, sm + 4 * gi, sync) : 0.0;
            if (lane == 0) (gi == 0 ? out->v_sum : gi == 1 ? out->p_out_sum : out->p_in_sum) = t;
            if (border > 0 && gi > 0) {  // the node counts (whole numbers: exact in any order)
                const double n = lanes_final_sum(part + 2 + gi, nch, 5, lane, sm + 4 * gi, sync);
                if (lane == 0) (gi == 1 ? out->cnt_out : out->cnt_in) = n;
            }
            if (threadIdx.x == 0) out->counter[0] = 0;
        }
    }
}

// ComputeDiv, src/NSBase.cxx:1958-2080
template <int G>
__global__ void __launch_bounds__(LANES *G, 8 / G)
    k_divergence(Grid g, Phys ph, SysView P, const double *__restrict__ u, const double *__restrict__ v,
                 const double *__restrict__ w, double *__restrict__ part, DiagOut *out) {
    __shared__ double s_div[CH], s_vel[CH], s_dv[CH], sm[16];
    __shared__ bool last;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const double idx = ph.idx, idy = ph.idy, idz = ph.idz;
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    for (int c = blockIdx.x; c < P.nchunks; c += gridDim.x) {
        const int rows = min(CH, P.n - c * CH);
#pragma unroll 1
        for (int m = 0; m < RPL / G; ++m) {
            const int q = lane + (gi * (RPL / G) + m) * LANES;
            if (q >= rows) break;
            int i, j, k, f;
            g.ijk(P.cell[c * CH + q], i, j, k);
            double div = 0, uu = 0, vv = 0, ww = 0, DV = 0;
            if (i > 0 && g.P(i - 1, j, k) > -1 && (f = g.U(i, j, k)) > -1) {
                div += -u[f] * idx; DV += -u[f]; uu += u[f] * 0.5;
            }
            if (i < nx - 1 && g.P(i + 1, j, k) > -1 && (f = g.U(i + 1, j, k)) > -1) {
                div += u[f] * idx; DV += u[f]; uu += u[f] * 0.5;
            }
            if (j > 0 && g.P(i, j - 1, k) > -1 && (f = g.V(i, j, k)) > -1) {
                div += -v[f] * idy; DV += -v[f]; vv += v[f] * 0.5;
            }
            if (j < ny - 1 && g.P(i, j + 1, k) > -1 && (f = g.V(i, j + 1, k)) > -1) {
                div += v[f] * idy; DV += v[f]; vv += v[f] * 0.5;
            }
            if (k > 0 && g.P(i, j, k - 1) > -1 && (f = g.W(i, j, k)) > -1) {
                div += -w[f] * idz; DV += -w[f]; ww += w[f] * 0.5;
            }
            if (k < nz - 1 && g.P(i, j, k + 1) > -1 && (f = g.W(i, j, k + 1)) > -1) {
                div += w[f] * idz; DV += w[f]; ww += w[f] * 0.5;
            }
            if (i == 0 && (f = g.U(i, j, k)) > -1) {
                div += -u[f] * idx; DV += -u[f]; uu += u[f] * 0.5;
            }
            if (i == nx - 1 && (f = g.U(i + 1, j, k)) > -1) {
                div += u[f] * idx; DV += u[f]; uu += u[f] * 0.5;
            }
            s_dv[q] = fabs(DV);
            s_div[q] = fabs(div);
            s_vel[q] = sqrt(uu * uu + vv * vv + ww * ww);
        }
        __syncthreads();
        const GroupSync sync{gi + 1};
        for (int j = gi; j < 2; j += G) {  // 0: sum of div^2 and its maximum, 1: sum of |u| and the maximum of DV
            double acc = 0.0, mx = 0.0;
            const double *val = j == 0 ? s_div : s_dv;
#pragma unroll
            for (int m = 0; m < RPL; ++m) {
                const int q = lane + m * LANES;
                if (q < rows) {
                    acc = j == 0 ? __fma_rn(s_div[q], s_div[q], acc) : acc + s_vel[q];
                    mx = dmaxv(mx, val[q]);
                }
            }
            const double sum = lanes_tree_sum<double>(acc, lane, sm + 4 * j, sync);
            const double ext = lanes_extreme<true>(mx, lane, sm + 8 + 4 * j, sync);
            if (lane == 0) {
                part[(size_t)c * 4 + j] = sum;
                part[(size_t)c * 4 + 3 - j] = ext;
            }
        }
        if (!last_block_arrive(&out->counter[1], (unsigned)P.nchunks, &last)) continue;
        for (int j = gi; j < 2; j += G) {
            const double sum = lanes_final_sum(part + j, P.nchunks, 4, lane, sm + 4 * j, sync);
            double mx = 0.0;
            for (int q = lane; q < P.nchunks; q += LANES) mx = dmaxv(mx, __ldcg(part + (size_t)q * 4 + 3 - j));
            mx = lanes_extreme<true>(mx, lane, sm + 8 + 4 * j, sync);
            if (lane == 0) {
                if (j == 0) {
                    out->sumdiv2 = sum;
                    out->maxdiv = mx;
                    out->counter[1] = 0;
                } else {
                    out->sumvel = sum;
                    out->maxdv = mx;
                }
            }
        }
    }
}

// CorrectPressureField, src/NSBase.cxx:2367-2380: max, min, |pc|^2, p += beta pc
template <int G>
__global__ void __launch_bounds__(LANES *G, 8 / G)
    k_correct_pressure(SysView P, const double *__restrict__ pc, double *__restrict__ p, double beta,
                       double *__restrict__ part, DiagOut *out) {
    __shared__ double s_x[CH], sm[12];
    __shared__ bool last;
    const int gi = threadIdx.x / LANES, lane = threadIdx.x % LANES;
    for (int c = blockIdx.x; c < P.nchunks; c += gridDim.x) {
        const int rows = min(CH, P.n - c * CH);
#pragma unroll
        for (int m = 0; m < RPL / G; ++m) {
            const int q = lane + (gi * (RPL / G) + m) * LANES, r = c * CH + q;
            if (q < rows) {
                const double x = pc[r];
                s_x[q] = x;
                p[r] = p[r] + beta * x;
            }
        }
        __syncthreads();
        const GroupSync sync{gi + 1};
        for (int j = gi; j < 2; j += G) {  // 0: sum of squares, 1: maximum and minimum
            if (j == 0) {
                const double sq = lanes_tree_sum<double>(lane_dot(s_x, s_x, lane, rows), lane, sm, sync);
                if (lane == 0) part[(size_t)c * 3 + 2] = sq;
            } else {
                double mx = -HUGE_VAL, mn = HUGE_VAL;
#pragma unroll
                for (int m = 0; m < RPL; ++m) {
                    const int q = lane + m * LANES;
                    if (q < rows) {
                        mx = dmaxv(mx, s_x[q]);
                        mn = dminv(mn, s_x[q]);
                    }
                }
                mx = lanes_extreme<true>(mx, lane, sm + 4, sync);
                mn = lanes_extreme<false>(mn, lane, sm + 8, sync);
                if (lane == 0) {
                    part[(size_t)c * 3 + 0] = mx;
                    part[(size_t)c * 3 + 1] = mn;
                }
            }
        }
        if (!last_block_arrive(&out->counter[2], (unsigned)P.nchunks, &last)) continue;
        for (int j = gi; j < 2; j += G) {
            if (j == 0) {
                const double sq = lanes_final_sum(part + 2, P.nchunks, 3, lane, sm, sync);
                if (lane == 0) {
                    out->pcsq = sq;
                    out->counter[2] = 0;
                }
            } else {
                double a = -HUGE_VAL, b = HUGE_VAL;
                for (int q = lane; q < P.nchunks; q += LANES) {
                    a = dmaxv(a, __ldcg(part + (size_t)q * 3 + 0));
                    b = dminv(b, __ldcg(part + (size_t)q * 3 + 1));
                }
                a = lanes_extreme<true>(a, lane, sm + 4, sync);
                b = lanes_extreme<false>(b, lane, sm + 8, sync);
                if (lane == 0) {
                    out->pcmax = a;
                    out->pcmin = b;
                }
            }
        }
    }
}

// Initpvector default profile, src/NSBase.cxx:2671-2681
__global__ void k_default_pressure(Grid g, SysView P, double p0, double p1, double *__restrict__ p) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < P.n; r += gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(P.cell[r], i, j, k);
        p[r] = (p1 - p0) * ((double)i + 1.0) / ((double)g.nx) + p0;
    }
}

__global__ void k_gather_image(const int *__restrict__ map, long ncells, const double *__restrict__ f,
                               double *__restrict__ img) {
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += (long)gridDim.x * blockDim.x) {
        int r = map[c];
        img[c] = r > -1 ? f[r] : 0.0;
    }
}
__global__ void k_scatter_image(const int *__restrict__ map, long ncells, const double *__restrict__ img,
                                double *__restrict__ f) {
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += (long)gridDim.x * blockDim.x) {
        int r = map[c];
        if (r != -1) f[r] = img[c];
    }
}

// FieldsToImage face averages, src/NSBase.cxx:425-466
__global__ void k_face_average(Grid g, const double *__restrict__ u, const double *__restrict__ v,
                               const double *__restrict__ w, double *__restrict__ out) {
    const long N = (long)g.nx * g.ny * g.nz;
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < N; c += (long)gridDim.x * blockDim.x) {
        int i, j, k;
        g.ijk(c, i, j, k);
        double au = 0, av = 0, aw = 0;
        int a = g.U(i + 1, j, k), b = g.U(i, j, k);
        if (a > -1 && b > -1) au = (u[a] + u[b]) * 0.50;
        else if (a > -1) au = (u[a]) * 0.50;
        else if (b > -1) au = (u[b]) * 0.50;
        b = g.V(i, j, k);
        if (j < g.ny - 1) {
            a = g.V(i, j + 1, k);
            if (a > -1 && b > -1) av = (v[a] + v[b]) * 0.50;
            else if (a > -1) av = (v[a]) * 0.50;
            else if (b > -1) av = (v[b]) * 0.50;
        } else if (b > -1) av = (v[b]) * 0.50;
        b = g.W(i, j, k);
        if (k < g.nz - 1) {
            a = g.W(i, j, k + 1);
            if (a > -1 && b > -1) aw = (w[a] + w[b]) * 0.50;
            else if (a > -1) aw = (w[a]) * 0.50;
            else if (b > -1) aw = (w[b]) * 0.50;
        } else if (b > -1) aw = (w[b]) * 0.50;
        out[3 * c + 0] = au;
        out[3 * c + 1] = av;
        out[3 * c + 2] = aw;
    }
}

// warm start of a pressure-drop sweep: u, v, w *= ratio; p = p0' + (p - p0) ratio
__global__ void k_scale_fields(double *u, int nu, double *v, int nv, double *w, int nw, double *p, int np,
                               double ratio, double p0_old, double p0_new) {
    const long total = (long)nu + nv + nw + np;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        if (i < nu) u[i] = u[i] * ratio;
        else if (i < (long)nu + nv) v[i - nu] = v[i - nu] * ratio;
        else if (i < (long)nu + nv + nw) w[i - nu - nv] = w[i - nu - nv] * ratio;
        else {
            const long k = i - nu - nv - nw;
            p[k] = p0_new + (p[k] - p0_old) * ratio;
        }
    }
}

// ---- launchers ---------------------------------------------------------------
static inline int rows_grid(long n) { return (int)std::max<long>(1, std::min<long>((n + 255) / 256, 152L * 16)); }
static inline int chunk_grid(int nch) { return std::max(1, std::min(nch, 152 * 8)); }

// schemefactor 0, and magnitudes for which no product of the momentum rows
// underflows where it would count (cross_face, own_face)
static bool plain_momentum(const Phys &ph) {
    for (double v : {ph.mu, ph.rho, ph.dx, ph.dy, ph.dz})
        if (!(v >= 1e-20 && v <= 1e20)) return false;
    return ph.schemefactor == 0;
}

template <bool PLAIN>
static void launch_mom(int comp, const Grid &g, const Phys &ph, const SysView &A, const double *uc, const double *vc,
                       const double *wc, cudaStream_t st) {
    count_launches(1);
    if (comp == 0) k_mom_x<PLAIN><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, uc, vc, wc);
    else if (comp == 1) k_mom_y<PLAIN><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, uc, vc, wc);
    else k_mom_z<PLAIN><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, uc, vc, wc);
}

void launch_assemble_momentum(int comp, const Grid &g, const Phys &ph, const SysView &A, const double *uc,
                              const double *vc, const double *wc, cudaStream_t st) {
    if (A.n <= 0) return;
    if (plain_momentum(ph)) launch_mom<true>(comp, g, ph, A, uc, vc, wc, st);
    else launch_mom<false>(comp, g, ph, A, uc, vc, wc, st);
}

void launch_momentum_rhs(int comp, const Grid &g, const Phys &ph, const SysView &A, const double *p,
                         const double *x, cudaStream_t st) {
    if (A.n <= 0) return;
    if (comp == 0) { count_launches(1); k_mom_rhs<0><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, x); }
    else if (comp == 1) { count_launches(1); k_mom_rhs<1><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, x); }
    else { count_launches(1); k_mom_rhs<2><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, x); }
}

void launch_hat(const SysView &A, const Phys &ph, const double *xc, const double *xold, double *hat,
                cudaStream_t st) {
    if (A.n <= 0) return;
    count_launches(1); k_hat<<<rows_grid(A.n), 256, 0, st>>>(A, ph, xc, xold, hat);
}

void launch_assemble_pressure(int mode, int relax, const Grid &g, const Phys &ph, const SysView &S,
                              const SysView &U, const SysView &V, const SysView &W, const double *uc,
                              const double *vc, const double *wc, const double *p, cudaStream_t st) {
    if (S.n <= 0) return;
    const double *au = (mode == 1) ? U.rowsum : U.coef;  // slot P is the first slot
    const double *av = (mode == 1) ? V.rowsum : V.coef;
    const double *aw = (mode == 1) ? W.rowsum : W.coef;
    count_launches(1); k_pressure<<<rows_grid(S.n), 256, 0, st>>>(mode, relax, g, ph, S, au, av, aw, uc, vc, wc, p);
}

void launch_correct_velocity(int comp, int simplec, const Grid &g, const Phys &ph, const SysView &A,
                             const double *pc, double *x, double dvmax, cudaStream_t st) {
    if (A.n <= 0) return;
    const double *den = simplec ? A.rowsum : A.coef;
    if (comp == 0) { count_launches(1); k_correct<0><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, den, pc, x, dvmax); }
    else if (comp == 1) { count_launches(1); k_correct<1><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, den, pc, x, dvmax); }
    else { count_launches(1); k_correct<2><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, den, pc, x, dvmax); }
}

void launch_correct_velocity_simpler(int comp, const Grid &g, const Phys &ph, const SysView &A, const double *p,
                                     const double *hat, double *x, double p_0, double p_1, cudaStream_t st) {
    if (A.n <= 0) return;
    if (comp == 0) { count_launches(1); k_correct_simpler<0><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, hat, x, p_0, p_1); }
    else if (comp == 1) { count_launches(1); k_correct_simpler<1><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, hat, x, p_0, p_1); }
    else { count_launches(1); k_correct_simpler<2><<<rows_grid(A.n), 256, 0, st>>>(g, ph, A, p, hat, x, p_0, p_1); }
}

void launch_scale_fields(double *u, int nu, double *v, int nv, double *w, int nw, double *p, int np, double ratio,
                         double p0_old, double p0_new, cudaStream_t st) {
    count_launches(1);
    k_scale_fields<<<152 * 8, 256, 0, st>>>(u, nu, v, nv, w, nw, p, np, ratio, p0_old, p0_new);
}

void launch_velocity_post(const double *temp, double *x, int n, const KState *st_dev, int limit, double dvmax,
                          cudaStream_t st) {
    if (n <= 0) return;
    count_launches(1); k_velocity_post<<<rows_grid(n), 256, 0, st>>>(temp, x, n, st_dev, limit, dvmax);
}

void launch_permeability(const Grid &g, const double *u, const double *p, int border, double *part, DiagOut *out,
                         cudaStream_t st) {
    long plane = (long)g.ny * g.nz;
    int nch = (int)((plane + CH - 1) / CH);
    count_launches(1); k_permeability<<<chunk_grid(nch), CH, 0, st>>>(g, u, p, border, part, out);
}

void launch_divergence(const Grid &g, const Phys &ph, const SysView &P, const double *u, const double *v,
                       const double *w, double *part, DiagOut *out, cudaStream_t st) {
    if (P.n <= 0) {
        cudaMemsetAsync(&out->maxdv, 0, 4 * sizeof(double), st);
        return;
    }
    count_launches(1);
    if (wide_chunks(P.nchunks, device_sm_count()))
        k_divergence<WIDE_G><<<chunk_grid(P.nchunks), LANES * WIDE_G, 0, st>>>(g, ph, P, u, v, w, part, out);
    else
        k_divergence<NARROW_G><<<chunk_grid(P.nchunks), LANES * NARROW_G, 0, st>>>(g, ph, P, u, v, w, part, out);
}

void launch_correct_pressure(const SysView &P, const double *pc, double *p, double beta, double *part,
                             DiagOut *out, cudaStream_t st) {
    if (P.n <= 0) return;
    count_launches(1);
    if (wide_chunks(P.nchunks, device_sm_count()))
        k_correct_pressure<WIDE_G><<<chunk_grid(P.nchunks), LANES * WIDE_G, 0, st>>>(P, pc, p, beta, part, out);
    else
        k_correct_pressure<NARROW_G><<<chunk_grid(P.nchunks), LANES * NARROW_G, 0, st>>>(P, pc, p, beta, part, out);
}

void launch_default_pressure(const Grid &g, const SysView &P, double p0, double p1, double *p, cudaStream_t st) {
    if (P.n <= 0) return;
    count_launches(1); k_default_pressure<<<rows_grid(P.n), 256, 0, st>>>(g, P, p0, p1, p);
}

void launch_gather_image(const int *map, long ncells, const double *field, double *img, cudaStream_t st) {
    count_launches(1); k_gather_image<<<rows_grid(ncells), 256, 0, st>>>(map, ncells, field, img);
}
void launch_scatter_image(const int *map, long ncells, const double *img, double *field, cudaStream_t st) {
    count_launches(1); k_scatter_image<<<rows_grid(ncells), 256, 0, st>>>(map, ncells, img, field);
}
void launch_face_average(const Grid &g, const double *u, const double *v, const double *w, double *vavg,
                         cudaStream_t st) {
    long N = (long)g.nx * g.ny * g.nz;
    count_launches(1); k_face_average<<<rows_grid(N), 256, 0, st>>>(g, u, v, w, vavg);
}

}  // namespace ns3d
