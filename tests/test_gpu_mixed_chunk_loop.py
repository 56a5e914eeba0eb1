"""The FP32 loop with resident chunks against the FP32 loops it replaces, bit
for bit, at the edges of its range: one chunk, a chunk and a row, the unit
counts at which its reduction tree gains a level (8, 16, 32 chunks are 32, 64
and 128 units), the largest set it takes on a 152-SM GPU and the first one it
leaves.

The other loops are reached by attaching the solver to a group of many lanes:
a lane's share of the SMs is then too small for resident chunks.  All loops
promise the same FP32 arithmetic in the same order, so the tolerance is zero.
"""
import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu

BOXES = [(16, 8, 8), (41, 5, 5), (16, 32, 16), (33, 16, 16), (32, 32, 16), (33, 32, 32), (152, 32, 32), (153, 32, 32),
         (1100, 1, 1)]


def _solve(lib, img, group, outer=2):
    s = solver(lib, img, params(lib, precision=capi.MIXED, maxitSIMPLE=outer, vsolvertol=1e-7, pcsolvertol=1e-7,
                                maxitsolver=60))
    if group:
        group.attach(s)
    r = s.solve()
    out = (r.K, r.it_u, r.it_v, r.it_w, r.it_p, r.krylov_iterations), s.fields()
    s.close()
    return out


@pytest.mark.parametrize("shape", BOXES)
def test_boxes_bitwise(gpulib, shape):
    img = np.zeros(shape, np.uint8)
    if shape[1] > 8:
        img[synth.random_image(shape, 0.97, 11) == 1] = 1
    own = _solve(gpulib, img, None)
    group = capi.Group(gpulib, lanes=16)
    try:
        other = _solve(gpulib, img, group)
    finally:
        group.destroy()
    assert own[0] == other[0]
    for a, b in zip(own[1], other[1]):
        assert np.array_equal(a, b)
