"""The five-phase FP32 loop gives the same bits every time, alone and beside
other solves: its last update of x and the conversion of x to FP64 have no grid
barrier between them, so both must be the same thread's.  One multilevel system
of several hundred chunks and one without a hierarchy (above 2^18 rows), solved
again and again from the same guess, on the whole GPU and on a share of it.
"""
import threading

import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _system(lib, img, precision):
    s = solver(lib, img, params(lib, precision=precision))
    rng = np.random.default_rng(5)
    n = s.sizes
    s.set_fields(1.0 + 1e-3 * rng.standard_normal(n.np), 1e-6 * rng.standard_normal(n.nu),
                 1e-6 * rng.standard_normal(n.nv), 1e-6 * rng.standard_normal(n.nw))
    s.assemble_momentum()
    s.assemble_pressure_correction(True)
    m = s.n(capi.SYS_P)
    x0, b = 1e-3 * rng.standard_normal(m), rng.standard_normal(m)

    def solve():
        x, info = s.solve_system(capi.SYS_P, x0, 1e-9, 400, rhs=b)
        return x, (info.iterations, info.info, info.error)
    return s, solve


@pytest.mark.parametrize("precision,shape,fluid", [(capi.MIXED_MG, (72, 70, 71), 0.95), (capi.MIXED, (66, 66, 66), 1.0)],
                         ids=["multilevel", "jacobi"])
def test_repeated_solves_have_the_same_bits(gpulib, precision, shape, fluid):
    s, solve = _system(gpulib, synth.random_image(shape, fluid, 13), precision)
    first, info = solve()
    bad = []
    for k in range(25):
        x, i = solve()
        if i != info or not np.array_equal(x, first):
            bad.append(("alone", k, i))
    stop = threading.Event()

    def run(seed):  # (ns3d_solve: while it runs, other solves take a share of the SMs)
        img = synth.random_image((48, 50, 46), 0.95, seed)
        while not stop.is_set():
            o = solver(gpulib, img, params(gpulib, precision=precision, maxitSIMPLE=3))
            o.solve()
            o.close()
    threads = [threading.Thread(target=run, args=(20 + k,)) for k in range(3)]
    for t in threads:
        t.start()
    try:
        for k in range(25):
            x, i = solve()
            if i != info or not np.array_equal(x, first):
                bad.append(("beside others", k, i))
    finally:
        stop.set()
        for t in threads:
            t.join()
    s.close()
    assert not bad
