"""The multilevel loop with packed columns (large systems): the same bits as
the loop of merged sets, which reads the table of columns.  Boxes on both sides
of its size limit, with the largest distance between columns that the packed
form holds (255 x 257 rows between planes) and one more (not packed), and a
porous image with isolated pores.  Both loops do the same arithmetic, so the
tolerance is zero.
"""
import numpy as np
import pytest

from helpers import params
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,fluid", [((80, 81, 80), 1.0), ((81, 81, 80), 1.0), ((9, 255, 257), 1.0),
                                         ((9, 256, 256), 1.0), ((84, 84, 84), 0.93)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "%g" % v)
def test_packed_equals_merged(gpulib, shape, fluid):
    img = synth.random_image(shape, fluid, 7)
    p = params(gpulib, method="SIMPLEC", precision=capi.MIXED_MG, maxitSIMPLE=2)
    raw = synth.to_raw(img)
    alone = capi.Solver(gpulib, p, raw, img.shape)
    ra, fa = alone.solve(), alone.fields()
    alone.close()
    pair = [capi.Solver(gpulib, p, raw, img.shape) for _ in range(2)]
    rc, st = capi.solve_lockstep(gpulib, pair)
    assert rc == 0 and not st.any(), gpulib.ns3d_last_error()
    for s in pair:
        r = s.result()
        assert r.krylov_iterations == ra.krylov_iterations and r.K == ra.K
        for a, b in zip(s.fields(), fa):
            assert np.array_equal(a, b)
        s.close()
