"""The split form's classical path: exponents and digits of both operands in one
launch (clusters over k), tiles as work units where the grid leaves SMs idle.
Bit-exact against the oracle over slice counts, formats and sizes around a
line group (16), a k tile (128), a k block and the chunk of a cluster's CTA;
with lines of zeros, of subnormal numbers and of a wide range; the
allocation-free call (whole tiles) and a batch give the same bits."""
import numpy as np
import pytest

from conftest import rand
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    return torch


def padded(x, pad):
    import torch
    m, n = x.shape
    big = torch.full((n, m + pad), float("nan"), dtype=torch.float64, device="cuda")
    big[:, :m] = to_dev(x).t()
    return big[:, :m].t()


def want_of(orc, A, B, C, s, alpha, beta, fmt):
    from oracle import coeffs as oc
    return orc.split_fmm_dgemm(oc.classical(), A, B, C.copy(order="F"), s, alpha, beta, fmt=fmt)


@pytest.mark.parametrize("m,n,k,s,fmt", [
    (1, 1, 1, 2, "bf16"), (15, 17, 63, 3, "bf16"), (16, 16, 128, 4, "bf16"), (17, 300, 129, 5, "bf16"),
    (129, 257, 64, 8, "bf16"), (130, 100, 65, 7, "bf16"), (300, 270, 450, 6, "bf16"), (40, 50, 1025, 6, "bf16"),
    (20, 700, 2049, 6, "bf16"), (70, 30, 9000, 5, "bf16"), (1030, 20, 300, 6, "bf16"), (64, 64, 16384, 8, "bf16"),
    (5, 9, 127, 2, "fp8"), (33, 260, 257, 7, "fp8"), (140, 300, 1000, 10, "fp8"), (60, 40, 5000, 12, "fp8"),
    (1100, 260, 128, 11, "fp8")])
@pytest.mark.parametrize("alpha,beta,pad", [(1.0, 1.0, 0), (-0.75, 0.0, 3), (2.0, 0.5, 16)])
def test_classical_bitexact(fmm, orc, torch_cuda, m, n, k, s, fmt, alpha, beta, pad):
    A, B, C = rand(m, k, 11), rand(k, n, 12), rand(m, n, 13)
    dC = padded(C, pad)
    fmm.split_dgemm(padded(A, pad), padded(B, pad), dC, None, 0, s, alpha=alpha, beta=beta, fmt=fmt)
    want = want_of(orc, A, B, C, s, alpha, beta, fmt)
    assert np.array_equal(to_host(dC), want)


@pytest.mark.parametrize("s,fmt", [(6, "bf16"), (8, "bf16"), (10, "fp8"), (12, "fp8")])
def test_unusual_lines_bitexact(fmm, orc, torch_cuda, s, fmt):
    m, n, k = 50, 40, 700
    A, B, C = rand(m, k, 21), rand(k, n, 22), rand(m, n, 23)
    A[3, :] = 0.0
    A[7, :] *= 2.0 ** -1040          # subnormal down to the low words
    A[8, :] = 0.0
    A[8, 5] = 5e-324
    A[9, :] *= 2.0 ** -1022
    A[20, ::2] *= 2.0 ** -200        # entries far below their line's maximum
    A[21, 699] = -(2.0 ** 500)
    B[:, 4] *= 2.0 ** 900
    B[:, 5] = 0.0
    B[:, 39] *= 2.0 ** -1030
    want = want_of(orc, A, B, C, s, 1.0, 1.0, fmt)
    dC = to_dev(C)
    fmm.split_dgemm(to_dev(A), to_dev(B), dC, None, 0, s, fmt=fmt)
    assert np.array_equal(to_host(dC), want)


@pytest.mark.parametrize("m,n,k", [(200, 300, 640), (1050, 70, 200), (31, 33, 3000)])
def test_whole_tiles_and_batches_give_the_same_bits(fmm, torch_cuda, m, n, k):
    import torch
    A, B, C = to_dev(rand(m, k, 31)), to_dev(rand(k, n, 32)), rand(m, n, 33)
    got = []
    dC = to_dev(C)
    fmm.split_dgemm(A, B, dC, None, 0, 6, alpha=-1.0, beta=0.5)
    got.append(to_host(dC))
    dC = to_dev(C)
    fmm.split_dgemm_noalloc(A, B, dC, None, 0, 6, alpha=-1.0, beta=0.5)
    got.append(to_host(dC))
    other = to_dev(rand(90, 80, 1)), to_dev(rand(80, 70, 2)), to_dev(rand(90, 70, 3))
    dC = to_dev(C)
    fmm.batch_dgemm([{"A": A, "B": B, "C": dC, "slices": 6, "alpha": -1.0, "beta": 0.5},
                     {"A": other[0], "B": other[1], "C": other[2], "slices": 7, "fmt": "fp8"}])
    got.append(to_host(dC))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    dC = to_dev(C)
    ws = torch.empty(fmm.split_workspace_size(m, n, k, None, 0, 6), dtype=torch.uint8, device="cuda")
    with torch.cuda.graph(graph):
        fmm.split_dgemm(A, B, dC, None, 0, 6, alpha=-1.0, beta=0.5, workspace=ws)
    dC.copy_(to_dev(C))
    graph.replay()
    torch.cuda.synchronize()
    got.append(to_host(dC))
    for g in got[1:]:
        assert np.array_equal(g, got[0])
