"""The FP64 BiCGSTAB loops at the edges of their ranges, bit for bit
against the CPU oracle.  One chunk per block: one row over a chunk, the chunk counts at which its
reduction trees lose or gain a level (32/33, 64/65, 128/129 chunks), the
largest set it takes on a 152-SM GPU and the first one it leaves to the
several-chunks-per-block loop, rows whose west or east entry directly precedes
or follows the diagonal, three systems in one launch, and the same through the
allocation-free entry point.  Both sides use one fixed floating-point contract,
so the tolerance is zero.
"""
import ctypes as C

import numpy as np
import pytest

from helpers import params, solver
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu

# all-fluid boxes of exactly 1024 k (+ 1) cells, a line of cells (W = row - 1,
# E = row + 1), and porous images
# (up to 36 and 76 chunks the loop splits a chunk over four and two blocks)
BOXES = [(16, 8, 8), (41, 5, 5), (36, 32, 32), (37, 32, 32), (75, 32, 32), (76, 32, 32), (77, 32, 32), (32, 32, 32), (33, 32, 32), (64, 32, 32), (65, 32, 32), (64, 64, 32), (43, 96, 32),
         (152, 32, 32), (153, 32, 32), (1100, 1, 1)]


def _systems(lib, img, sys):
    s = solver(lib, img, params(lib, alpha=0.7))
    rng = np.random.default_rng(3)
    n = s.sizes
    s.set_fields(1.0 + 1e-3 * rng.standard_normal(n.np), 1e-6 * rng.standard_normal(n.nu),
                 1e-6 * rng.standard_normal(n.nv), 1e-6 * rng.standard_normal(n.nw))
    s.assemble_momentum()
    s.assemble_pressure_correction(True)
    m = s.n(sys)
    x, info = s.solve_system(sys, 1e-3 * rng.standard_normal(m), 1e-11, 12, rhs=rng.standard_normal(m))
    coef, nbr, rhs, _ = s.system(sys)
    s.close()
    return x, (info.iterations, info.info, info.error), (coef, nbr)


# the largest set and the first one beyond it of the loops with several chunks
# per block: two chunks (four groups each), four, eight, any number on 152 SMs;
# and columns more than 65535 rows away
SEVERAL = [(304, 32, 32), (305, 32, 32), (608, 32, 32), (609, 32, 32), (1216, 32, 32), (1217, 32, 32), (3, 264, 256)]


@pytest.mark.parametrize("shape", BOXES + SEVERAL)
def test_boxes_bitwise(gpulib, oracle, shape):
    img = np.zeros(shape, np.uint8)
    for sys in (capi.SYS_P, capi.SYS_U):
        g, o = _systems(gpulib, img, sys), _systems(oracle, img, sys)
        assert np.array_equal(g[0], o[0]) and g[1] == o[1]


@pytest.mark.parametrize("shape,seed", [((23, 19, 29), 1), ((47, 31, 37), 2)])
def test_three_systems_in_one_launch(gpulib, oracle, shape, seed):
    """A momentum solve (u, v, w of 11 to 45 chunks each, together at most 152)
    and the following pressure correction, as one outer iteration runs them."""
    img = synth.random_image(shape, 0.9, seed)
    out = []
    for lib in (gpulib, oracle):
        s = solver(lib, img, params(lib, alpha=0.7, maxitSIMPLE=2))
        r = s.solve()
        out.append((r.K, r.it_u, r.it_v, r.it_w, r.it_p, r.krylov_iterations, s.fields()))
        s.close()
    assert out[0][:6] == out[1][:6]
    for a, b in zip(out[0][6], out[1][6]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("edge", [3, 16, 40])
def test_noalloc_bitwise(gpulib, edge):
    torch = pytest.importorskip("torch")
    img = synth.random_image((edge, edge, edge), 0.95, 7)
    x_ref, info_ref, (coef, nbr) = _systems(gpulib, img, capi.SYS_P)
    rng = np.random.default_rng(3)
    s = solver(gpulib, img, params(gpulib, alpha=0.7))
    n = s.sizes
    for m in (n.np, n.nu, n.nv, n.nw):
        rng.standard_normal(m)  # the draws of _systems' fields
    s.close()
    m = coef.shape[1]
    npad = (m + 1023) // 1024 * 1024 + 1024
    pad = lambda a, v: np.concatenate([a, np.full(a.shape[:-1] + (npad - m,), v, a.dtype)], -1)
    x0, b = 1e-3 * rng.standard_normal(m), rng.standard_normal(m)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pad(coef, 0.0), pad(nbr, -1), pad(b, 0.0),
                                                                      pad(x0, 0.0))]
    f = gpulib.ns3d_bicgstab_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p] * 4 + [C.c_int32, C.c_int32, C.c_double, C.c_int32, C.c_void_p, C.POINTER(capi.SolveInfo)]
    info = capi.SolveInfo()
    assert f(*[t.data_ptr() for t in dev], m, npad, 1e-11, 12, torch.cuda.current_stream().cuda_stream,
             C.byref(info)) == 0
    assert np.array_equal(dev[3].cpu().numpy()[:m], x_ref)
    assert (info.iterations, info.info, info.error) == info_ref
