"""The split form's Z digit planes and C updates at the edges of their tiles:
bit-exact against the oracle for sub-block counts up to the shared-memory
form's 64 and beyond it, product groups of one (beta applied once), rows and
columns around a tile of 32..256 rows x 4 columns, every plane count, and the
largest level sums a carry can meet."""
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


@pytest.mark.parametrize("alg,levels,m,n,k,s,fmt", [
    ("222", 3, 41, 70, 35, 6, "bf16"),      # 64 sub-blocks: the widest shared-memory form, uneven sub-blocks
    ("322", 2, 97, 35, 30, 5, "bf16"),      # 36 sub-blocks
    ("444", 2, 35, 50, 40, 4, "bf16"),      # 256 sub-blocks: one thread row per sub-block
    ("444", 2, 70, 33, 40, 11, "fp8"),
    ("222", 1, 515, 13, 300, 8, "bf16"),    # 258-row product grid, 7-column last group
    ("232", 1, 130, 259, 260, 12, "fp8"),   # all seven FP8 planes, three levels above G
    ("333", 1, 100, 101, 60, 8, "bf16"),    # k_pad 64: levels 3 and 2 share the high plane
    ("222", 1, 66, 65, 90, 2, "fp8"),       # no digit plane at all
    ("322", 1, 200, 67, 40, 7, "fp8"),      # 6 and
    ("232", 2, 260, 31, 50, 6, "bf16"),     # 16 sub-blocks: four and two columns per thread
])
@pytest.mark.parametrize("alpha,beta", [(1.0, 1.0), (-0.75, 0.5), (2.0, 0.0)])
@pytest.mark.parametrize("groups", ["one", "several"])
def test_c_updates_bitexact(fmm, orc, algs, torch_cuda, alg, levels, m, n, k, s, fmt, alpha, beta, groups):
    import torch

    from oracle import coeffs as oc
    A, B, C = rand(m, k, 21), rand(k, n, 22), rand(m, n, 23)
    f = fmm.new_fmm(COEFFS / f"{alg}.txt")
    try:
        need = fmm.split_workspace_size(m, n, k, f, levels, s, fmt)
        ws = torch.empty(need if groups == "one" else need // 3, dtype=torch.uint8, device="cuda")
        dC = to_dev(C)
        fmm.split_dgemm(to_dev(A), to_dev(B), dC, f, levels, s, alpha=alpha, beta=beta, workspace=ws, fmt=fmt)
        got = to_host(dC)
    finally:
        fmm.free_fmm(f)
    want = orc.split_fmm_dgemm(oc.power(algs[alg], levels), A, B, C.copy(order="F"), s, alpha, beta, fmt=fmt)
    assert np.array_equal(got, want), float(np.max(np.abs(got - want)))


@pytest.mark.parametrize("s,fmt", [(6, "bf16"), (8, "bf16"), (12, "fp8")])
def test_largest_level_sums(fmm, orc, torch_cuda, s, fmt):
    """k = 16384, every operand near the top of its digit range and of one sign"""
    from oracle import coeffs as oc
    v = 1.0 - 2.0 ** -9 - 2.0 ** -17 - 2.0 ** -25
    A, B = np.full((24, 16384), -v, order="F"), np.full((16384, 20), v, order="F")
    C = np.zeros((24, 20), order="F")
    dC = to_dev(C)
    fmm.split_dgemm(to_dev(A), to_dev(B), dC, None, 0, s, fmt=fmt)
    want = orc.split_fmm_dgemm(oc.classical(), A, B, C.copy(order="F"), s, fmt=fmt)
    assert np.array_equal(to_host(dC), want)


@pytest.mark.parametrize("alg,levels", [(None, 0), ("222", 1)])
@pytest.mark.parametrize("s,fmt", [(6, "bf16"), (7, "bf16"), (8, "bf16"), (11, "fp8"), (12, "fp8")])
def test_digits_around_the_last_unit(fmm, orc, algs, torch_cuda, alg, levels, s, fmt):
    """elements from the last digit's unit to far below it, of both signs: the
    large element that sets a row's exponent meets zeros of B"""
    from oracle import coeffs as oc
    m, n, k = 64, 20, 40
    A, B, C = rand(m, k, 31), rand(k, n, 32), np.zeros((m, n), order="F")
    A *= 2.0 ** -(np.arange(m, dtype=np.float64)[:, None] % 32 + 38)
    A[::3, 1::4] = 2.0 ** -(np.arange(0, m, 3, dtype=np.float64)[:, None] % 32 + 38)   # ties among them
    A[:, [0, k // 2]] = 0.75
    B[[0, k // 2], :] = 0.0
    f = fmm.new_fmm(COEFFS / f"{alg}.txt") if alg else None
    try:
        dC = to_dev(C)
        fmm.split_dgemm(to_dev(A), to_dev(B), dC, f, levels, s, fmt=fmt)
    finally:
        if f is not None:
            fmm.free_fmm(f)
    want = orc.split_fmm_dgemm(oc.power(algs[alg], levels) if alg else oc.classical(), A, B, C.copy(order="F"), s, fmt=fmt)
    assert np.array_equal(to_host(dC), want)
