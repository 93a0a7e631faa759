"""A call whose temporary is the process's first, inside a stream capture."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import torch, fmm_blis_gb300 as fmm
def R(r, c): return torch.rand((c, r), device="cuda", dtype=torch.float64).t()
f = fmm.strassen_fmm()
fmm.dgemm(R(97, 45), R(45, 61), R(97, 61), f, 1)          # tables and attributes; needs no temporary
A, B, C = R(1024, 1000), R(1000, 1024), R(1024, 1024)
D = C.clone()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    fmm.dgemm(A, B, C, f, 1)
graph.replay()
fmm.dgemm(A, B, D, f, 1)
torch.cuda.synchronize()
assert torch.equal(C, D) and fmm.take_device_error() == 0
print("same bits")
"""


def test_first_temporary_inside_a_capture(fmm):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same bits" in r.stdout, r.stderr[-2000:]
