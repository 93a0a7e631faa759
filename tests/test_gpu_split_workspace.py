"""The split form at the limits of its caller's workspace."""
import numpy as np
import pytest

from conftest import COEFFS, rand
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

FMM_ERR_WORKSPACE = 9


def least_workspace(m, n, k, mt, kt, nt, s):
    """one FP8 product: maxima, exponents, digit slices and 8 bytes of level
    accumulators per element, each rounded up to 256 bytes"""
    def pad(x, to):
        return -(-x // to) * to

    me, ne, ke = -(-m // mt), -(-n // nt), -(-k // kt)
    m_pad, n_pad, k_pad = pad(me, 256 if me >= 1024 else 128), pad(ne, 256), pad(ke, 128)
    parts = [8 * kt * m, 8 * kt * n, 4, 4 * m_pad, 4 * n_pad, s * m_pad * k_pad, s * n_pad * k_pad, 8 * m_pad * n_pad]
    return sum(pad(p, 256) for p in parts)


@pytest.mark.parametrize("alg,levels,m,n,k,s", [
    (None, 0, 64, 64, 64, 7), (None, 0, 300, 270, 450, 9), (None, 0, 1100, 260, 128, 12), (None, 0, 2600, 2050, 200, 10),
    ("222", 1, 515, 300, 260, 8), ("232", 2, 260, 310, 250, 11)])
@pytest.mark.parametrize("way", ["call", "batch"])
def test_fp8_least_workspace(fmm, alg, levels, m, n, k, s, way):
    import torch
    f = fmm.new_fmm(COEFFS / f"{alg}.txt") if alg else None
    mt, kt, nt = (f.m_tilde ** levels, f.k_tilde ** levels, f.n_tilde ** levels) if alg else (1, 1, 1)
    A, B, C = to_dev(rand(m, k, 41)), to_dev(rand(k, n, 42)), rand(m, n, 43)
    want = to_dev(C)
    fmm.split_dgemm(A, B, want, f, levels, s, alpha=-0.75, beta=0.5, fmt="fp8")
    least = least_workspace(m, n, k, mt, kt, nt, s)
    for nbytes, accepted in ((least, True), (least - 256, False)):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        dC = to_dev(C)
        try:
            if way == "call":
                fmm.split_dgemm(A, B, dC, f, levels, s, alpha=-0.75, beta=0.5, workspace=ws, fmt="fp8")
            else:
                fmm.batch_dgemm([{"A": A, "B": B, "C": dC, "fmm": f, "levels": levels, "slices": s, "fmt": "fp8",
                                  "alpha": -0.75, "beta": 0.5}], workspace=ws)
        except fmm.FmmError as e:
            assert not accepted and e.status == FMM_ERR_WORKSPACE
            continue
        assert accepted
        assert np.array_equal(to_host(dC), to_host(want))
    assert fmm.take_device_error() == 0


MEM_ALLOC, MEM_FREE = 10, 11   # CU_GRAPH_NODE_TYPE_MEM_ALLOC, _MEM_FREE


@pytest.mark.parametrize("m,n,k,s,fmt", [(300, 700, 450, 6, "bf16"), (64, 64, 64, 7, "bf16"), (1100, 260, 300, 9, "fp8"),
                                         (128, 128, 16384, 6, "bf16")])
@pytest.mark.parametrize("full", [False, True])
def test_captured_call_holds_no_allocation(fmm, m, n, k, s, fmt, full):
    """A captured classical call on the caller's workspace is a graph without
    allocation nodes, so it can be cloned and have two executables at a time;
    both give the plain call's bits."""
    import ctypes

    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    A, B, C = to_dev(rand(m, k, 51)), to_dev(rand(k, n, 52)), rand(m, n, 53)
    want = to_dev(C)
    fmm.split_dgemm(A, B, want, None, 0, s, alpha=-0.75, beta=0.5, fmt=fmt)
    ws = torch.empty(fmm.split_workspace_size(m, n, k, None, 0, s, fmt, full=full), dtype=torch.uint8, device="cuda")
    dC = to_dev(C)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    h, graph = ctypes.c_void_p(st.cuda_stream), ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(h, 2) == 0   # CU_STREAM_CAPTURE_MODE_RELAXED
    try:
        fmm.split_dgemm(A, B, dC, None, 0, s, alpha=-0.75, beta=0.5, workspace=ws, stream=st, fmt=fmt)
    finally:
        assert cu.cuStreamEndCapture(h, ctypes.byref(graph)) == 0
    count = ctypes.c_size_t()
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    kinds = []
    for x in nodes:
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(x), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    assert kinds and MEM_ALLOC not in kinds and MEM_FREE not in kinds
    clone = ctypes.c_void_p()
    assert cu.cuGraphClone(ctypes.byref(clone), graph) == 0
    execs = []
    for g in (graph, clone, graph):
        e = ctypes.c_void_p()
        assert cu.cuGraphInstantiateWithFlags(ctypes.byref(e), g, ctypes.c_ulonglong(0)) == 0
        execs.append(e)
    for e in execs:
        dC.copy_(to_dev(C))
        torch.cuda.synchronize()
        assert cu.cuGraphLaunch(e, h) == 0
        st.synchronize()
        assert np.array_equal(to_host(dC), to_host(want))
        assert cu.cuGraphExecDestroy(e) == 0
    assert cu.cuGraphDestroy(graph) == 0 and cu.cuGraphDestroy(clone) == 0
    assert fmm.take_device_error() == 0
