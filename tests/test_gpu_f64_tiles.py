"""The plain FP64 form's tiles at their edges: every pipelined tile (64 x 64,
16 x 8, 8 x 8 by the size of the product grid), the one-launch small FMM
problems, k below, at and past a copy
step and the stages of the ring, sub-arrays with odd leading dimensions, the
cluster path's two tiles; against the oracle within the FP64 bound, and the
batched call (64, 32 and 16 wide items) bit for bit against the single calls."""
import numpy as np
import pytest

from conftest import C_BOUND, COEFFS, fmm_bound, rand
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    return torch


def sub(x, pad):
    """x as the top rows of a larger column-major device array"""
    import torch
    m, n = x.shape
    big = torch.full((n, m + pad), float("nan"), dtype=torch.float64, device="cuda")
    big[:, :m] = to_dev(x).t()
    return big[:, :m].t()


@pytest.mark.parametrize("m,n,k,alg,levels", [
    (1, 1, 1, None, 0), (8, 8, 16, None, 0), (9, 17, 15, None, 0), (130, 65, 17, None, 0), (129, 300, 48, None, 0),
    (500, 520, 63, None, 0), (1300, 1290, 64, None, 0), (2049, 700, 65, None, 0), (5000, 9, 31, None, 0),
    (40, 3000, 100, None, 0), (300, 299, 301, "222", 1), (700, 640, 33, "333", 1), (1100, 1030, 128, "222", 1),
    (257, 258, 130, "444", 1), (260, 200, 190, "232", 2), (50, 60, 3, "322", 1),
    (97, 61, 45, "222", 1), (3, 13, 7, "222", 1), (16, 16, 32, "222", 1), (17, 200, 35, "333", 1),
    (100, 90, 81, "444", 1), (130, 120, 150, "322", 1), (40, 44, 130, "222", 2),
    (128, 128, 4096, None, 0), (65, 7, 2050, None, 0), (257, 129, 1300, None, 0), (310, 320, 900, None, 0)])
@pytest.mark.parametrize("alpha,beta,pad", [(1.0, 1.0, 0), (-0.5, 0.0, 3), (2.0, 0.25, 8)])
def test_tiles_match_oracle(fmm, orc, algs, torch_cuda, m, n, k, alg, levels, alpha, beta, pad):
    from oracle import coeffs as oc
    A, B, C = rand(m, k, 31), rand(k, n, 32), rand(m, n, 33)
    dA, dB, dC = sub(A, pad), sub(B, pad), sub(C, pad)
    f = fmm.new_fmm(COEFFS / f"{alg}.txt") if alg else None
    try:
        fmm.dgemm(dA, dB, dC, f, levels, alpha=alpha, beta=beta)
        got = to_host(dC)
    finally:
        if f is not None:
            fmm.free_fmm(f)
    if alg:
        want = orc.fmm_dgemm(oc.power(algs[alg], levels), A, B, C.copy(order="F"), alpha=alpha, beta=beta)
    else:
        want = orc.dgemm(A, B, C.copy(order="F"), alpha, beta)
    bound = fmm_bound(alpha * A, B, beta * C, k, C_BOUND[(alg, levels)] if alg else 2)
    assert np.max(np.abs(got - want)) <= bound
    if pad:   # nothing outside the operand was written
        whole = dC.t().as_strided((n, m + pad), (m + pad, 1))
        assert bool(whole[:, m:].isnan().all())


def test_infinities_and_nans_stay_where_they_belong(fmm, torch_cuda):
    """a non-finite entry reaches its own row or column only, whatever lies past the tile edges"""
    m, n, k = 70, 45, 50
    A, B, C = rand(m, k, 41), rand(k, n, 42), rand(m, n, 43)
    A[69, 3], B[4, 44] = np.inf, np.nan
    dC = to_dev(C)
    fmm.dgemm(to_dev(A), to_dev(B), dC, None, 0)
    got = to_host(dC)
    assert np.isfinite(got[:69, :44]).all()
    assert not np.isfinite(got[69, :]).any() and np.isnan(got[:, 44]).all()


@pytest.mark.parametrize("sizes", ["one_deep", "even", "many_small"])
def test_batch_items_give_single_call_bits(fmm, torch_cuda, sizes):
    import torch
    f2, f3 = fmm.new_fmm(COEFFS / "222.txt"), fmm.new_fmm(COEFFS / "333.txt")
    shapes = {"one_deep": [(200, 180, 2100, f2, 1), (30, 40, 20, None, 0), (65, 33, 90, f3, 1)],
              "even": [(300 + 7 * i, 280 - 5 * i, 200 + i, (None, f2, f3)[i % 3], int(i % 3 > 0)) for i in range(9)],
              "many_small": [(1 + 13 * i, 90 - i, 5 + 3 * i, (None, f2)[i % 2], i % 2) for i in range(40)]}[sizes]
    try:
        probs, want = [], []
        for i, (m, n, k, f, L) in enumerate(shapes):
            A, B, C0 = to_dev(rand(m, k, 700 + i)), to_dev(rand(k, n, 750 + i)), rand(m, n, 800 + i)
            beta = (1.0, 0.0, 0.5)[i % 3]
            dC = to_dev(C0)
            fmm.dgemm(A, B, dC, f, L, alpha=-1.5, beta=beta)
            want.append(to_host(dC))
            probs.append({"A": A, "B": B, "C": to_dev(C0), "fmm": f, "levels": L, "slices": 0, "alpha": -1.5,
                          "beta": beta})
        fmm.batch_dgemm(probs)
        torch.cuda.synchronize()
        for i, p in enumerate(probs):
            assert np.array_equal(to_host(p["C"]), want[i]), f"problem {i}"
    finally:
        fmm.free_fmm(f2)
        fmm.free_fmm(f3)
