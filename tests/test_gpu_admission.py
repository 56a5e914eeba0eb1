"""The server's footprint estimate counts what a multilevel mixed-precision
request holds (FP32 copies of its systems and the hierarchy), so a budget that
has room for one such request does not admit two.  And the estimate is an upper
bound of what a solve of an all-fluid image takes from the device.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import params
from ns3d_gb300 import capi, synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPE = (96, 64, 64)
FP64_BYTES = (SHAPE[0] + 1) * SHAPE[1] * SHAPE[2] * 816 + (64 << 20)  # the estimate of an FP64 request


def test_budget_for_one_multilevel_request_admits_one(gpulib):
    raw = synth.to_raw(np.zeros(SHAPE, np.uint8))
    p = params(gpulib, precision=capi.MIXED_MG, maxitSIMPLE=20, simpletol=1e-12)
    srv = capi.Server(gpulib, max_active=2, hbm_budget_bytes=int(2.02 * FP64_BYTES))
    tickets = [srv.submit(p, raw, SHAPE) for _ in range(2)]
    for t in tickets:
        srv.wait(t)
    st = srv.stats()
    srv.stop()
    assert st.completed == 2 and st.peak_active == 1


CHILD = r'''
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import numpy as np, torch
import ns3d_gb300
from ns3d_gb300 import capi
from helpers import params, solver
lib = ns3d_gb300.lib()
mode, shape = int(sys.argv[2]), tuple(int(v) for v in sys.argv[3].split("x"))
w = solver(lib, np.zeros((8, 8, 8), np.uint8), params(lib, precision=mode, maxitSIMPLE=1))
w.solve()
free = torch.cuda.mem_get_info()[0]
s = solver(lib, np.zeros(shape, np.uint8), params(lib, precision=mode, maxitSIMPLE=2))
s.solve()
print("TOOK", free - torch.cuda.mem_get_info()[0])
'''


@pytest.mark.parametrize("mode,per_cell", [(capi.FP64, 816), (capi.MIXED, 816 + 4 * 76), (capi.MIXED_MG, 816 + 4 * 76 + 48)])
def test_estimate_bounds_what_a_solve_takes(gpulib, mode, per_cell):
    pytest.importorskip("torch")
    shape = (150, 97, 101)
    out = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(mode), "x".join(map(str, shape))],
                         stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert out.returncode == 0 and "TOOK" in out.stdout, out.stdout
    took = int(out.stdout.split("TOOK")[1])
    assert took <= (shape[0] + 1) * shape[1] * shape[2] * per_cell + (64 << 20)
    print(mode, took / np.prod(shape))
