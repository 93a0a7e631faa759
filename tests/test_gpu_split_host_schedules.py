"""The host-buffer split call's schedules and its refusals."""
import time

import numpy as np
import pytest

from conftest import COEFFS, rand
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    return torch


def test_refused_call_copies_nothing(fmm, torch_cuda):
    """k beyond the split form's 16384 per product: refused before the
    operands go up, 17 MB that a call of nearly the same size copies."""
    def call(k):
        A, B, C = np.ones((64, k), order="F"), np.ones((k, 64), order="F"), np.zeros((64, 64), order="F")
        st, best = None, float("inf")
        for _ in range(5):
            t0 = time.perf_counter()
            st = fmm.lib().fmm_gpu_split_strassen_ab_ex(1.0, A.ctypes.data, 64, B.ctypes.data, k, 1.0, C.ctypes.data,
                                                        64, 64, 64, k, fmm.FmmT(), 0, 6, 0)
            best = min(best, time.perf_counter() - t0)
        return st, best

    st, accepted = call(16384)
    assert st == 0
    st, refused = call(16384 + 64)
    assert st not in (0, 1) and refused < accepted / 10
    assert fmm.take_device_error() == 0


def alg_of(fmm, name):
    return fmm.new_fmm(COEFFS / f"{name}.txt") if name else None


# (algorithm, levels, m, n, k, slices, format, GEMM launches): operands beyond the sizes that go without overlap
SCHEDULES = [
    (None, 0, 2560, 8001, 100, 6, "bf16", 8),     # 2 x 4 blocks of pair tiles
    ("222", 1, 2067, 5801, 300, 9, "fp8", 8),     # 2 x 4, uneven halves and parts
    ("222", 1, 1501, 8003, 200, 6, "bf16", 8),    # 2 x 4 of single-SM tiles
    ("222", 1, 250, 22401, 200, 5, "bf16", 4),    # 1 x 4: one tile row
    (None, 0, 9001, 250, 600, 6, "bf16", 2),      # 2 x 1: one tile column
    (None, 0, 128, 2000, 2501, 7, "bf16", 2),     # 1 x 2
    ("222", 1, 2101, 2050, 2300, 6, "bf16", 4),   # 2 x 2
    (None, 0, 128, 256, 16000, 10, "fp8", 1),     # no blocks: a single tile, C in column chunks
    ("333", 2, 360, 361, 26000, 4, "bf16", 1),    # no blocks, C updates per sub-block
    ("322", 2, 7901, 7900, 64, 4, "bf16", 8),     # 36 sub-blocks in blocks
    ("222", 3, 10501, 10500, 64, 3, "bf16", 8),   # 64
]


@pytest.mark.parametrize("alpha,beta", [(1.0, 1.0), (-0.75, 0.5), (2.0, 0.0)])
@pytest.mark.parametrize("alg,levels,m,n,k,s,fmt,launches", SCHEDULES)
def test_schedules_equal_device_call(fmm, torch_cuda, alg, levels, m, n, k, s, fmt, launches, alpha, beta):
    """Every schedule, by its number of GEMM launches, gives the device call's
    bits, writes C's own elements only and, with beta 0, reads none of them;
    leading dimensions larger than the row counts."""
    f = alg_of(fmm, alg)
    A, B, C = rand(m, k, 61), rand(k, n, 62), rand(m, n, 63)
    Ab, Bb, Cb = (np.full((x.shape[0] + p, x.shape[1]), 7.0, order="F") for x, p in ((A, 3), (B, 5), (C, 7)))
    Ab[:m], Bb[:k], Cb[:m] = A, B, C if beta != 0.0 else np.nan
    dC = to_dev(C)
    fmm.split_dgemm(to_dev(A), to_dev(B), dC, f, levels, s, alpha=alpha, beta=beta, fmt=fmt)
    want = to_host(dC)
    fmm.read_kernel_timing()
    fmm.set_kernel_timing(True)
    try:
        st = fmm.lib().fmm_gpu_split_strassen_ab_ex(
            alpha, Ab.ctypes.data, m + 3, Bb.ctypes.data, k + 5, beta, Cb.ctypes.data, m + 7, m, n, k,
            f if f is not None else fmm.FmmT(), levels, s, 1 if fmt == "fp8" else 0)
        _, ran, _ = fmm.read_kernel_timing()
    finally:
        fmm.set_kernel_timing(False)
    assert st == 0 and (ran == launches if levels < 3 else ran >= launches)
    assert np.array_equal(Cb[:m], want)
    assert np.all(Cb[m:] == 7.0)
    assert fmm.take_device_error() == 0
