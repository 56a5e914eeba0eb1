"""ns3d_bicgstab_noalloc takes all the device memory it needs in its first call,
whatever the sizes of the later ones.  Which kernels a call runs depends on its
size, and CUDA loads a kernel's code when it is first used, so the first call
has to load them all.  A process of its own, in which nothing has been loaded:
one chunk, then 30 (split over four blocks), 60 (over two) and 64; the device's
free memory stays what it was after the first call.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from ns3d_gb300 import capi
import ns3d_gb300
lib = ns3d_gb300.lib()
f = lib.ns3d_bicgstab_noalloc
f.restype = C.c_int
f.argtypes = [C.c_void_p] * 4 + [C.c_int32, C.c_int32, C.c_double, C.c_int32, C.c_void_p, C.POINTER(capi.SolveInfo)]


def system(n):
    """A line of cells: the neighbours W and E are the rows before and after."""
    coef, nbr = np.zeros((7, n)), np.full((6, n), -1, np.int32)
    coef[0] = 2.5
    coef[1], coef[2] = -1.0, -1.0
    nbr[0, 1:], nbr[1, :-1] = np.arange(n - 1), np.arange(1, n)
    b = np.random.default_rng(n).standard_normal(n)
    return [torch.from_numpy(a).cuda() for a in (coef, nbr, b, np.zeros(n))]


systems = [(n, system(n)) for n in (1024, 30 * 1024, 60 * 1024, 64 * 1024, 1024)]
torch.cuda.synchronize()
free = []
for n, dev in systems:
    info = capi.SolveInfo()
    rc = f(*[t.data_ptr() for t in dev], n, n, 1e-10, 40, torch.cuda.current_stream().cuda_stream, C.byref(info))
    assert rc == 0, (n, rc)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
    print(n, info.iterations, info.info, free[-1])
print("SAME" if len(set(free)) == 1 else "CHANGED")
'''


def test_free_memory_is_the_same_after_every_call(gpulib):
    pytest.importorskip("torch")
    out = subprocess.run([sys.executable, "-c", CHILD, ROOT], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                         timeout=300, env=dict(os.environ, CUDA_MODULE_LOADING="LAZY"))
    assert out.returncode == 0 and out.stdout.strip().endswith("SAME"), out.stdout
