"""A bounded wait that runs out, in each of the loop kernels: the call returns
NS3D_ERR_TIMEOUT, and the next solve on the same handle gives the bits of a
fresh one.  The wait limit is short and set for the one call only; nothing
faults or hangs (ns3d_debug_barrier_timeout).  The sizes pick the kernel on 152
SMs: a chunk split over four and two blocks, a chunk per block, two, four, eight
and more chunks per block in FP64; the three FP32 loops, the multilevel one with
its columns unpacked and packed.

`extra` 2 (a chunk split over a cluster) lets only the first block of each
cluster give up on the partials: the others go on to the next hand-over of
operands, and the first one has to outlast their stores.
"""
import ctypes

import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi

pytestmark = pytest.mark.gpu

CASES = [(capi.FP64, (20, 32, 32), 1), (capi.FP64, (20, 32, 32), 2), (capi.FP64, (16, 8, 8), 2),
         (capi.FP64, (64, 32, 32), 1), (capi.FP64, (64, 32, 32), 2), (capi.FP64, (100, 32, 32), 1),
         (capi.FP64, (300, 32, 32), 1), (capi.FP64, (600, 32, 32), 1), (capi.FP64, (1200, 32, 32), 1),
         (capi.FP64, (1300, 32, 32), 1),
         (capi.MIXED, (100, 32, 32), 1), (capi.MIXED, (200, 32, 32), 1), (capi.MIXED, (300, 32, 32), 1),
         (capi.MIXED_MG, (70, 70, 70), 1), (capi.MIXED_MG, (600, 32, 32), 1)]


@pytest.mark.parametrize("precision,shape,extra", CASES,
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_timeout_is_reported_and_recovered(gpulib, precision, shape, extra):
    hook = gpulib.ns3d_debug_barrier_timeout
    hook.restype, hook.argtypes = ctypes.c_int, [ctypes.c_int32, ctypes.c_double]
    img = np.zeros(shape, np.uint8)
    rng = np.random.default_rng(8)
    n = img.size
    x0, b = 1e-3 * rng.standard_normal(n), rng.standard_normal(n)
    out = []
    for fail in (True, False):
        s = solver(gpulib, img, params(gpulib, precision=precision, alpha=0.7))
        s.assemble_momentum()
        s.assemble_pressure_correction(True)
        solve = lambda: s.solve_system(capi.SYS_P, x0, 1e-6, 30, rhs=b)
        if fail:
            try:
                assert hook(extra, 0.02) == 0
                with pytest.raises(capi.NS3DError) as e:
                    solve()
            finally:
                assert hook(0, 0.0) == 0
            assert e.value.code == capi.ERR_TIMEOUT
            assert b"timed out" in gpulib.ns3d_last_error()
        x, info = solve()
        out.append((x, info.iterations, info.info, info.error))
        s.close()
    assert out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])
