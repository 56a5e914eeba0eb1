"""The device-built aggregation hierarchy of the multilevel mixed solves on
odd, thin and tiny boxes: the pressure solve meets its FP64 residual test,
takes far fewer inner iterations than with Jacobi, and repeats bit for bit.

Bound: the solver stops when |b - A x|^2 <= tol^2 |b|^2 in FP64; recomputing
the residual in another summation order moves it by at most about 16 eps
|A||x| per row, below 1e-3 of tol |b| at tol = 1e-8 on these systems.
"""
import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu
TOL = 1e-8


def _solve(lib, shape, phi, seed, precision):
    s = solver(lib, synth.random_image(shape, phi, seed), params(lib, precision=precision, alpha=0.7))
    s.assemble_momentum()
    s.assemble_pressure_correction(True)
    coef, nbr, _, _ = s.system(capi.SYS_P)
    n = s.n(capi.SYS_P)
    rhs = np.random.default_rng(seed).standard_normal(n)
    x, info = s.solve_system(capi.SYS_P, np.zeros(n), TOL, 2000, rhs=rhs)
    s.close()
    cols = np.where(nbr >= 0, nbr, np.arange(n))
    ax = coef[0] * x + (coef[1:] * x[cols]).sum(0)
    return n, x, info, np.linalg.norm(rhs - ax) / np.linalg.norm(rhs)


# one coarse level just above the coarsest size, odd extents, flat and thin
# boxes, blocks cut by the far faces, and more blocks than one scan tile
@pytest.mark.parametrize("shape", [(9, 9, 8), (17, 13, 11), (2, 33, 47), (65, 3, 31), (31, 29, 2), (37, 41, 39)])
def test_hierarchy_shapes(gpulib, shape):
    n, x, info, res = _solve(gpulib, shape, 0.97, 5, capi.MIXED_MG)
    assert n > 512 and info.info == capi.SUCCESS and res <= TOL * 1.001
    _, x2, info2, _ = _solve(gpulib, shape, 0.97, 5, capi.MIXED_MG)
    assert np.array_equal(x, x2) and info.iterations == info2.iterations
    _, _, jac, _ = _solve(gpulib, shape, 0.97, 5, capi.MIXED)
    assert info.iterations < jac.iterations
