"""The FP32 loops without a hierarchy against a CPU restatement of a whole
mixed-precision solve (tests/cpp/mixed_restatement.cpp), bit for bit: one
chunk, a chunk and a row, the unit counts at which the reduction tree of the
resident-chunk loop gains a level (8, 16, 32 chunks are 32, 64, 128 units), its
largest set on 152 SMs, the first set of the three-phase loop and the first of
the five-phase loop (above 2^18 rows).  Both sides round every operation and
add in one fixed order, so the tolerance is zero.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INNER_TOL, INNER_CAP = 1e-4, 400  # MixedSet's defaults


@pytest.fixture(scope="module")
def restatement(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("mixed") / "restatement.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(ROOT, "tests", "cpp", "mixed_restatement.cpp"), "-o", so], check=True)
    f = C.CDLL(so).mixed_restatement
    d, i = C.POINTER(C.c_double), C.POINTER(C.c_int)
    f.restype, f.argtypes = None, [d, i, d, d, C.c_int, C.c_double, C.c_int, C.c_double, C.c_int, i, i, d]

    def solve(coef, nbr, b, x0, tol, maxit):
        x = x0.copy()
        its, info, err = C.c_int(), C.c_int(), C.c_double()
        arr = [np.ascontiguousarray(coef, np.float64), np.ascontiguousarray(nbr, np.int32),
               np.ascontiguousarray(b, np.float64)]
        f(arr[0].ctypes.data_as(d), arr[1].ctypes.data_as(i), arr[2].ctypes.data_as(d), x.ctypes.data_as(d), len(x), tol,
          maxit, INNER_TOL, INNER_CAP, C.byref(its), C.byref(info), C.byref(err))
        return x, (its.value, info.value, err.value)
    return solve


def _system(lib, img, sys, **kw):
    s = solver(lib, img, params(lib, alpha=0.7, **kw))
    rng = np.random.default_rng(3)
    n = s.sizes
    s.set_fields(1.0 + 1e-3 * rng.standard_normal(n.np), 1e-6 * rng.standard_normal(n.nu),
                 1e-6 * rng.standard_normal(n.nv), 1e-6 * rng.standard_normal(n.nw))
    s.assemble_momentum()
    s.assemble_pressure_correction(True)
    m = s.n(sys)
    return s, 1e-3 * rng.standard_normal(m), rng.standard_normal(m)


def test_restatement_solves_the_system(oracle, restatement):
    """On the CPU: the restated solve meets its tolerance, measured by numpy."""
    s, x0, b = _system(oracle, synth.random_image((14, 13, 12), 0.9, 4), capi.SYS_P)
    coef, nbr, _, _ = s.system(capi.SYS_P)
    s.close()
    tol = 1e-9
    x, (its, info, err) = restatement(coef, nbr, b, x0, tol, 2000)
    ax = coef[0] * x
    for k in range(6):
        m = nbr[k] >= 0
        ax[m] += coef[k + 1][m] * x[nbr[k][m]]
    assert info == 0 and 0 < its < 2000 and err <= tol
    assert abs(np.linalg.norm(b - ax) / np.linalg.norm(b) - err) <= 1e-3 * tol


CASES = [((16, 8, 8), 1.0), ((41, 5, 5), 1.0), ((16, 32, 16), 0.97), ((33, 16, 16), 1.0), ((32, 32, 16), 1.0),
         ((33, 32, 32), 0.97), ((1100, 1, 1), 1.0), ((152, 32, 32), 1.0), ((153, 32, 32), 1.0), ((257, 32, 32), 1.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("sys", [capi.SYS_P, capi.SYS_U], ids=["pressure", "momentum"])
@pytest.mark.parametrize("shape,fluid", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "%g" % v)
def test_loops_equal_the_restatement(gpulib, restatement, shape, fluid, sys):
    s, x0, b = _system(gpulib, synth.random_image(shape, fluid, 11), sys, precision=capi.MIXED)
    coef, nbr, _, _ = s.system(sys)
    for tol, maxit in ((1e-10, 45), (1e-3, 200)):
        x, info = s.solve_system(sys, x0, tol, maxit, rhs=b)
        xr, ir = restatement(coef, nbr, b, x0, tol, maxit)
        assert (info.iterations, info.info, info.error) == ir
        assert np.array_equal(x, xr)
    s.close()
