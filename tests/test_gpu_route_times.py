"""Calls whose cost depends on which kernel form or tile a rule picks for them:
each takes no longer than a bound between the times of the right and the wrong
pick (best of several, events on the device), so a rule that moves them to the
wrong one shows."""
import pytest

from conftest import COEFFS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    return torch


def operand(torch, rows, cols):
    return (torch.rand((cols, rows), device="cuda", dtype=torch.float64) * 2 - 1).t()


def device_us(torch, f, reps=5, calls=4):
    for _ in range(2):
        f()
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(calls):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / calls * 1e3)
    return best


def test_c_updates_of_many_sub_blocks(fmm, torch_cuda):
    """Three Strassen levels on an 8 x 110 product grid: 64 C sub-blocks, 343
    products. About 250 us with a C update per sub-block, 530 us with all
    sub-blocks of an element in one thread."""
    m, n, k = 64, 880, 384
    f = fmm.new_fmm(COEFFS / "222.txt")
    A, B, C = operand(torch_cuda, m, k), operand(torch_cuda, k, n), operand(torch_cuda, m, n)
    ws = torch_cuda.empty(fmm.split_workspace_size(m, n, k, f, 3, 6), dtype=torch_cuda.uint8, device="cuda")
    assert device_us(torch_cuda, lambda: fmm.split_dgemm(A, B, C, f, 3, 6, 1.0, 0.5, ws)) < 400


def test_batch_of_unlike_c_updates(fmm, torch_cuda):
    """A problem of 36 sub-blocks and 121 products beside a classical one:
    about 300 us as a batch, 830 us with both in one C update launch whose
    blocks are shared out by tiles."""
    torch = torch_cuda
    f = fmm.new_fmm(COEFFS / "322.txt")
    ps = [{"A": operand(torch, m, k), "B": operand(torch, k, n), "C": operand(torch, m, n), "fmm": g, "levels": lv,
           "slices": s, "fmt": fmt}
          for m, n, k, g, lv, s, fmt in [(963, 267, 134, f, 2, 11, "fp8"), (675, 2091, 595, None, 0, 4, "bf16")]]
    b = fmm.make_batch(ps)
    ws = torch.empty(fmm.batch_workspace_size(b), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.batch_dgemm(b, workspace=ws)) < 550


def test_batch_of_unlike_small_c_updates(fmm, torch_cuda):
    """16 and 36 sub-blocks of small product grids beside classical problems:
    1360 us with one C update launch for all, shared out by tiles."""
    torch = torch_cuda
    f2, f3 = fmm.new_fmm(COEFFS / "222.txt"), fmm.new_fmm(COEFFS / "322.txt")
    ps = [{"A": operand(torch, m, k), "B": operand(torch, k, n), "C": operand(torch, m, n), "fmm": g, "levels": lv,
           "slices": s, "fmt": fmt}
          for m, n, k, g, lv, s, fmt in [(1069, 935, 147, None, 0, 7, "fp8"), (787, 293, 450, f2, 2, 8, "bf16"),
                                         (607, 1440, 524, None, 0, 12, "fp8"), (121, 123, 122, None, 0, 3, "bf16"),
                                         (484, 504, 46, f3, 2, 6, "fp8")]]
    b = fmm.make_batch(ps)
    ws = torch.empty(fmm.batch_workspace_size(b), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.batch_dgemm(b, workspace=ws)) < 900


@pytest.mark.parametrize("alg,shapes,bound", [
    ("222", [(2048, 2048, 2048, 1)], 15000),                    # tiles of 32: 13.6 ms; of 64 15.2, of 16 16.6
    ("232", [(1912, 2475, 97, 1), (169, 242, 116, 0)], 1800),   # tiles of 64: 1.5 ms; of 16 2.0
    ("222", [(512, 512, 512, 1)], 450),                         # tiles of 16: 0.32 ms; of 32 0.59, of 64 2.0
    ("333", [(1380, 185, 323, 1), (534, 382, 1340, 0)], 1200),  # unlike items on tiles of 16: 0.78 ms; of 32 1.7
])
def test_fp64_batch_tiles(fmm, torch_cuda, alg, shapes, bound):
    torch = torch_cuda
    f = fmm.new_fmm(COEFFS / f"{alg}.txt")
    ps = [{"A": operand(torch, m, k), "B": operand(torch, k, n), "C": operand(torch, m, n), "fmm": f if lv else None,
           "levels": lv, "slices": 0} for m, n, k, lv in shapes]
    b = fmm.make_batch(ps)
    ws = torch.empty(max(fmm.batch_workspace_size(b), 256), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.batch_dgemm(b, workspace=ws)) < bound


def test_c_updates_of_narrow_product_grids(fmm, torch_cuda):
    """256 sub-blocks, an 8 x 600 product grid: 5.2 ms with a block's threads
    on all of a tile's columns, 8.5 ms with 128 rows x 4 columns a block."""
    torch = torch_cuda
    m, n, k = 128, 9600, 768
    f = fmm.new_fmm(COEFFS / "444.txt")
    A, B, C = operand(torch, m, k), operand(torch, k, n), operand(torch, m, n)
    ws = torch.empty(fmm.split_workspace_size(m, n, k, f, 2, 6), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.split_dgemm(A, B, C, f, 2, 6, 1.0, 0.5, ws), reps=3, calls=2) < 7000


def test_c_updates_of_fp8_digits(fmm, torch_cuda):
    """81 sub-blocks of a 345 x 250 product grid in the FP8 format: 1.40 ms,
    1.59 ms with the Z digits put together one by one."""
    torch = torch_cuda
    m, n, k = 3101, 2244, 73
    f = fmm.new_fmm(COEFFS / "333.txt")
    A, B, C = operand(torch, m, k), operand(torch, k, n), operand(torch, m, n)
    ws = torch.empty(fmm.split_workspace_size(m, n, k, f, 2, 5, "fp8"), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.split_dgemm(A, B, C, f, 2, 5, 1.0, 0.0, ws, fmt="fp8")) < 1500


@pytest.mark.parametrize("s", range(2, 13))
@pytest.mark.parametrize("alg,levels,m,n,k", [(None, 0, 130, 70, 90), ("222", 1, 70, 45, 40), ("333", 1, 50, 61, 30),
                                              ("322", 2, 40, 37, 20)])
def test_fp8_digit_planes_bitexact(fmm, orc, algs, alg, levels, m, n, k, s):
    """every number of digit planes, in each form of the C update"""
    import numpy as np

    from conftest import rand
    from gpu_util import to_dev, to_host
    from oracle import coeffs as oc
    A, B, C = rand(m, k, 71), rand(k, n, 72), rand(m, n, 73)
    f = fmm.new_fmm(COEFFS / f"{alg}.txt") if alg else None
    plan = oc.power(algs[alg], levels) if alg else oc.classical()
    want = orc.split_fmm_dgemm(plan, A, B, C.copy(order="F"), s, -0.75, 0.5, fmt="fp8")
    dC = to_dev(C)
    fmm.batch_dgemm([{"A": to_dev(A), "B": to_dev(B), "C": dC, "fmm": f, "levels": levels, "slices": s, "fmt": "fp8",
                      "alpha": -0.75, "beta": 0.5}])
    assert np.array_equal(to_host(dC), want)
    dC = to_dev(C)
    fmm.split_dgemm(to_dev(A), to_dev(B), dC, f, levels, s, alpha=-0.75, beta=0.5, fmt="fp8")
    assert np.array_equal(to_host(dC), want)


def test_batch_of_long_and_short_c_updates(fmm, torch_cuda):
    """121 products of a 414 x 492 product grid beside four small problems:
    700 us with its C updates by sub-block, 770 in one launch with the others,
    whose blocks push its last ones into a second round."""
    torch = torch_cuda
    algs = {a: fmm.new_fmm(COEFFS / f"{a}.txt") for a in ("232", "333")}
    ps = [{"A": operand(torch, m, k), "B": operand(torch, k, n), "C": operand(torch, m, n), "fmm": algs.get(a), "levels": lv,
           "slices": s, "fmt": fmt, "beta": 0.5}
          for m, n, k, a, lv, s, fmt in [(45, 832, 36, "232", 2, 7, "fp8"), (50, 734, 124, "333", 1, 10, "fp8"),
                                         (159, 353, 160, "232", 1, 3, "bf16"), (1654, 1967, 276, "232", 2, 4, "bf16"),
                                         (65, 221, 2192, None, 0, 6, "bf16")]]
    b = fmm.make_batch(ps)
    ws = torch.empty(fmm.batch_workspace_size(b), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.batch_dgemm(b, workspace=ws)) < 740


def test_c_updates_of_many_products_on_small_grids(fmm, torch_cuda):
    """121 products, 16 sub-blocks, an 8 x 110 product grid: 96 us with a C
    update per sub-block, 168 with all products in one thread's chain."""
    torch = torch_cuda
    m, n, k = 32, 440, 432
    f = fmm.new_fmm(COEFFS / "232.txt")
    A, B, C = operand(torch, m, k), operand(torch, k, n), operand(torch, m, n)
    ws = torch.empty(fmm.split_workspace_size(m, n, k, f, 2, 6), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.split_dgemm(A, B, C, f, 2, 6, 1.0, 0.5, ws)) < 135


def test_batch_of_many_small_c_updates(fmm, torch_cuda):
    """20 problems of a handful of C update blocks: 145 us with one launch for
    all of them, 203 with one each."""
    torch = torch_cuda
    f = fmm.new_fmm(COEFFS / "333.txt")
    ps = [{"A": operand(torch, 33, 90), "B": operand(torch, 90, 101), "C": operand(torch, 33, 101), "fmm": f, "levels": 1,
           "slices": 3} for _ in range(20)]
    b = fmm.make_batch(ps)
    ws = torch.empty(fmm.batch_workspace_size(b), dtype=torch.uint8, device="cuda")
    assert device_us(torch, lambda: fmm.batch_dgemm(b, workspace=ws)) < 175


@pytest.mark.parametrize("kinds", [
    [("322", 2), ("222", 3), ("444", 2), ("333", 2)],                         # by sub-block, in one launch
    [("322", 2), (None, 0), ("222", 1), ("232", 2), ("333", 1)],              # each kind once
    [("222", 1), ("322", 1), ("222", 2), (None, 0), (None, 0), ("232", 2)],
])
@pytest.mark.parametrize("big", [False, True])
def test_batch_c_update_forms_equal_single_calls(fmm, torch_cuda, kinds, big):
    """every kind of C update launch of a batch, small product grids and some
    above two blocks per SM, gives the single calls' bits"""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(5)

    def rnd(r, c):
        return (torch.rand((c, r), generator=g, device="cuda", dtype=torch.float64) * 2 - 1).t()

    probs, want = [], []
    for i, (a, lv) in enumerate(kinds * 2):
        f = fmm.new_fmm(COEFFS / f"{a}.txt") if a else None
        m, n, k = (1500 + 61 * i, 1300 + 37 * i, 90) if big and i % 3 == 0 else (130 + 17 * i, 97 + 29 * i, 70 + 13 * i)
        p = {"A": rnd(m, k), "B": rnd(k, n), "C": rnd(m, n), "fmm": f, "levels": lv, "slices": 3 + i % 5,
             "fmt": "fp8" if i % 2 else "bf16", "alpha": -0.75, "beta": [1.0, 0.5, 0.0][i % 3]}
        c = p["C"].clone()
        fmm.split_dgemm(p["A"], p["B"], c, f, lv, p["slices"], alpha=p["alpha"], beta=p["beta"], fmt=p["fmt"])
        probs.append(p)
        want.append(c)
    fmm.batch_dgemm(probs)
    torch.cuda.synchronize()
    for i, (p, w) in enumerate(zip(probs, want)):
        assert torch.equal(p["C"], w), f"problem {i}"
    assert fmm.take_device_error() == 0
