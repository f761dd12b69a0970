"""The checks of caller CSR arrays (sixteen entries at a time): a bad row pointer, column or value is
found wherever it stands in stretches of 1 to 9,000 entries, and sound arrays pass."""
import numpy as np
import pytest


def _check(A, C, V, cols):
    from simplefem_gb300 import _native
    st = _native.gpu().feec_csr_check(len(A) - 1, cols, np.asarray(A, np.int32), np.asarray(C, np.int32),
                                      np.asarray(V, np.float64))
    return st == _native.FEEC_OK


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4096, 4097, 9000])
def test_csr_check_finds_every_bad_entry(n):
    rng = np.random.default_rng(n)
    cols = 50
    A = np.concatenate([[0], np.sort(rng.integers(0, n + 1, n - 1)), [n]])
    C, V = rng.integers(0, cols, n), rng.standard_normal(n)
    assert _check(A, C, V, cols)
    for k in {0, n // 2, n - 1, min(n - 1, 4095), min(n - 1, 4096)}:
        for bad in (-1, -2**31, cols, 2**31 - 1):
            D = C.copy()
            D[k] = bad
            assert not _check(A, D, V, cols), (k, bad)
        for bad in (np.nan, np.inf, -np.inf):
            W = V.copy()
            W[k] = bad
            assert not _check(A, C, W, cols), (k, bad)
        for good in (np.finfo(np.float64).max, -np.finfo(np.float64).max, 5e-324, -0.0):
            W = V.copy()
            W[k] = good
            assert _check(A, C, W, cols), (k, good)
        if k > 0:
            B = A.copy()
            B[k] = B[k + 1] + 1
            assert not _check(B, C, V, cols), k


def test_csr_check_extremes():
    big = 2**31 - 1
    assert _check([0, 1], [big - 1], [1.0], big) and not _check([0, 1], [big], [1.0], big)
    assert not _check([0, 1], [0], [1.0], 0)          # no column at all
    assert _check([0, 0], [], [], 0)
    assert not _check([1, 1], [0], [1.0], 1)
    # a fall whose difference overflows 32 bits
    assert not _check([0, 2 * 10**9, -2 * 10**9], [0, 0], [1.0, 1.0], 1)
