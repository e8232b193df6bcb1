"""Calls that read results back fail on a stream under capture: with an error
code, as any call, not with the end of the process (their device arrays are
given up while the failure unwinds)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes as C, os, sys
sys.path.insert(0, "tests")
import numpy as np, torch
import omega_h_v1_b200 as G
from conftest import build_gpu
rt = C.CDLL("libcudart.so.12")
L = G.lib()
m = build_gpu(24, size=0.03)     # (arrays above and below the size that is kept)
st = torch.cuda.Stream()
L.osh_b200_set_stream(m.h, C.c_void_p(st.cuda_stream))
G.check()
ne, nv, nt = m.count(1), m.count(0), m.count(3)
u = lambda n: np.zeros(n, np.uint32)
f = lambda n: np.zeros(n, np.float64)
calls = {
    "refine": lambda: L.osh_b200_refine_sets(m.h, 0.0, u(ne), u(ne), f(ne), u(ne)),
    "coarsen": lambda: L.osh_b200_coarsen_sets(m.h, 0.0, 1 / 3., u(ne), u(ne), u(ne), f(2 * ne),
                                               u(nv), f(nv), u(nv), u(nv)),
    "write": lambda: L.osh_write_vtk(m.h, sys.argv[2].encode()),
}
run = calls[sys.argv[1]]
run()                            # (derives what the call needs)
G.check()
torch.cuda.synchronize()
assert rt.cudaStreamBeginCapture(C.c_void_p(st.cuda_stream), 2) == 0
run()
print("error", L.osh_b200_last_error())
sys.stdout.flush()
os._exit(0)                      # the capture ends with the process, unused
"""


@pytest.mark.parametrize("call", ["refine", "coarsen", "write"])
def test_error_under_capture(call, tmp_path):
    r = subprocess.run([sys.executable, "-c", PROGRAM, call, str(tmp_path / "m.vtu")], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    assert r.stdout.startswith("error ") and r.stdout.strip() != "error 0", r.stdout
