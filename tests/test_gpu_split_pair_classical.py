"""CTA-pair tiles of classical problems: whole tiles, as calls without a
temporary (and batches) run them where a single call would cut the tiles of so
small a grid into work units. Bit-exact against the oracle."""
import numpy as np
import pytest

from conftest import rand
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1100, 700, 300), (1024, 256, 64), (1025, 257, 129)])
def test_pair_tiles_without_temporary(fmm, orc, m, n, k):
    from oracle import coeffs as oc
    A, B, C = rand(m, k, 401), rand(k, n, 402), rand(m, n, 403)
    dC = to_dev(C)
    fmm.split_dgemm_noalloc(to_dev(A), to_dev(B), dC, None, 0, 6, alpha=0.75, beta=-0.5)
    want = orc.split_fmm_dgemm(oc.classical(), A, B, C.copy(order="F"), 6, 0.75, -0.5)
    assert np.array_equal(to_host(dC), want)
    assert fmm.take_device_error() == 0


@pytest.mark.parametrize("fmt,s", [("bf16", 5), ("fp8", 9)])
def test_pair_tiles_in_a_batch(fmm, orc, fmt, s):
    from oracle import coeffs as oc
    m, n, k = 1100, 700, 300
    A, B, C = rand(m, k, 404), rand(k, n, 405), rand(m, n, 406)
    dC = to_dev(C)
    fmm.batch_dgemm([{"A": to_dev(A), "B": to_dev(B), "C": dC, "slices": s, "fmt": fmt, "alpha": 0.75, "beta": -0.5}])
    want = orc.split_fmm_dgemm(oc.classical(), A, B, C.copy(order="F"), s, 0.75, -0.5, fmt=fmt)
    assert np.array_equal(to_host(dC), want)
    assert fmm.take_device_error() == 0
