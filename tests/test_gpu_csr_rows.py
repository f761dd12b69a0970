"""The per-row exchange sort of sums and products where its packed words can go wrong: rows of 0, 1
and about 32, 512, 1024 and 2048 entries, columns whose span just fits beside the slot and the flag
and just does not, equal columns that merge, cancel and merge again, zeros. Bit-identical to the
oracle's serial sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_rows(rng, lengths, cols, span, zeros):
    A = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    C, V = [], []
    for k in lengths:
        lo = int(rng.integers(0, cols - span + 1))
        c = rng.integers(0, span, k)
        if k > 1:                            # both ends of the span are there
            c[0], c[-1] = span - 1, 0
        C.append(lo + c)
        v = rng.choice([1.0, -1.0, 0.3, -0.3, 1e9, 1e-9], k) if k % 2 else rng.standard_normal(k)
        v[rng.random(k) < zeros] = 0.0
        V.append(v)
    return A, np.concatenate(C).astype(np.int32), np.concatenate(V)


@pytest.mark.parametrize("span", [1, 3, 40, 700, 2**16, 2**20 - 1, 2**20, 2**21 - 2, 2**21 - 1, 2**22])
def test_rows_of_a_sum_match_serial_sort(cuda, span):
    import simplefem_gb300 as S
    from oracle import oracle
    rng = np.random.default_rng(span)
    l1 = [0, 1, 1, 16, 31, 32, 33, 255, 256, 500, 512, 513, 1000, 1023, 1024, 1500, 2047]
    l2 = [0, 0, 1, 15, 1, 1, 2, 256, 256, 12, 0, 0, 23, 0, 1, 548, 2]
    cols = span + 1000
    A1, C1, V1 = _random_rows(rng, l1, cols, span, 0.1)
    A2, C2, V2 = _random_rows(rng, l2, cols, span, 0.1)
    X, Y = S.MatrixCSR(len(l1), cols, A1, C1, V1), S.MatrixCSR(len(l2), cols, A2, C2, V2)
    for s1, s2 in ((1.0, 1.0), (0.7, -1.3), (1.0, 0.0)):
        M = S.MatrixCSRAddition(X, Y, s1, s2)
        A, C, V = oracle.csr_add(A1, C1, V1, A2, C2, V2, s1, s2)
        assert np.array_equal(M.A, A) and np.array_equal(M.C, C), (s1, s2)
        assert np.array_equal(M.V.view(np.int64), np.asarray(V, np.float64).view(np.int64)), (s1, s2)
