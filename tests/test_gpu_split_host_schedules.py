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
