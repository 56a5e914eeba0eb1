"""Momentum rows, bit for bit against the CPU oracle, where the short form of
the face terms meets its limits: zero, tiny and huge velocities of either sign,
overflowing fluxes, and physical constants on both sides of its ranges.  Both sides
evaluate the same expressions, so the tolerance is zero (NaN equals NaN).
"""
import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, -0.0, 5e-324, -1e-310, 1e-250, -1e-201, 1e-199, -1e-100, 1e-30, -1e10, 1e150, -1e199, 1e201, -1e250]
HUGE = [1.7e308, -1.7e308]  # sums and fluxes overflow to infinities and NaN


@pytest.mark.parametrize("shape", [(12, 11, 10), (9, 14, 1)])
@pytest.mark.parametrize("values", [[], SPECIAL, SPECIAL + HUGE], ids=["ordinary", "special", "huge"])
@pytest.mark.parametrize("kw", [dict(), dict(alpha=1.0), dict(mu=1e-22), dict(mu=1e-19, rho=1e19), dict(rho=3e20),
                                dict(dx=1e-21), dict(dx=1e-19, dy=1e-18, dz=1e19)],
                         ids=lambda k: "-".join("%s%g" % i for i in k.items()) or "default")
def test_momentum_rows(gpulib, oracle, shape, values, kw):
    img = synth.random_image(shape, 0.8, 5)
    g, o = solver(gpulib, img, params(gpulib, **kw)), solver(oracle, img, params(oracle, **kw))
    rng = np.random.default_rng(9)

    def velocity(n):
        f = 1e-6 * rng.standard_normal(n)
        pick = rng.random(n) < (0.5 if values else 0.0)
        if values:
            f[pick] = rng.choice(values, int(pick.sum()))
        return f

    n = g.sizes
    f = (1.0 + 1e-3 * rng.standard_normal(n.np), velocity(n.nu), velocity(n.nv), velocity(n.nw))
    for s in (g, o):
        s.set_fields(*f)
        s.assemble_momentum()
    for sys in (capi.SYS_U, capi.SYS_V, capi.SYS_W)[:3 if n.nw else 2]:
        for a, b in zip(g.system(sys), o.system(sys)):
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), sys
