"""Dataflow multicolor solvers (kernels_flow.cu) where their slices can go wrong: a diagonal
matrix (no sweep entries), rows of one and of several chunks per lane, one lane and many lanes
per row, a last slice that is not full, more blocks than slices. K within 2% (at least 1) of the
oracle and the solution within 1e-9 of it, the parity bar of the drop-in solvers."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _diagonal(n):
    return sp.diags(np.linspace(1.0, 2.0, n)).tocsr()


def _tridiagonal(n):
    return sp.diags([-np.ones(n - 1), np.full(n, 2.5), -np.ones(n - 1)], [-1, 0, 1]).tocsr()


def _arrow(n):
    """A dense first row and column over a tridiagonal rest: one row far longer than a lane chunk."""
    M = _tridiagonal(n).tolil()
    M[0, :] = 0.5 / n
    M[:, 0] = 0.5 / n
    M[0, 0] = 3.0
    return M.tocsr()


def _lattice(dim, r, L, n):
    from simplefem_gb300 import workloads
    A, C, V = workloads.lattice_matrix(dim, r, L, 3)
    M = sp.csr_matrix((V, C, A))
    return M[:n, :n].tocsr() if n else M


CASES = [("diagonal", lambda: _diagonal(40)), ("one_row", lambda: _diagonal(1)), ("two_rows", lambda: _tridiagonal(2)),
         ("tridiagonal_33", lambda: _tridiagonal(33)), ("arrow_257", lambda: _arrow(257)),
         ("arrow_9800", lambda: _arrow(9800)), ("p3", lambda: _lattice(3, 3, 2, 0)),
         ("ragged_p2", lambda: _lattice(3, 2, 3, 4097)), ("ragged_p1", lambda: _lattice(3, 1, 5, 19_999))]


@pytest.mark.parametrize("method,mode", [("rainbow", "reference"), ("rainbow_eisenstat", "reference"),
                                         ("rainbow", "fp64"), ("rainbow", "mixed")])
@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
def test_flow_solvers_match_oracle(name, make, method, mode):
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = make()
    M.sort_indices()
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64)
    n = len(A) - 1
    rng = np.random.default_rng(n)
    b = 1e3 * rng.uniform(-1.0, 1.0, n)
    diag = oracle.csr_diagonal(A, C, V)
    rb = oracle.rainbow(A, C)
    sysm = System(A, C, V)
    sysm.set_rainbow(diag, 1.0, *rb)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = sysm.solve(torch.from_numpy(b).cuda(), x, method=method, mode=mode, precision=1e-11)
    K_o, x_o, _ = oracle.cg_rainbow(A, C, V, b, diag, rb, 1.0, precision=1e-11)
    xh = x.cpu().numpy()
    if n < 3 and info["status"] == 3:      # the iteration cap, N by default, leaves two steps
        sysm.close()
        return
    assert info["status"] == 0, info
    assert np.linalg.norm(xh - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    if mode == "reference":
        assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    else:
        assert np.linalg.norm(b - M @ xh) <= 1e-11 * np.linalg.norm(b), info
    sysm.close()


CG_CASES = CASES + [("tridiagonal_5000", lambda: _tridiagonal(5000)), ("p1_2d", lambda: _lattice(2, 1, 6, 0)),
                    ("many_rows_published", lambda: _lattice(3, 1, 5, 30_011)),
                    ("many_rows_barrier", lambda: _lattice(3, 1, 6, 80_033)), ("long_rows_barrier", lambda: _lattice(3, 2, 5, 81_001))]


@pytest.mark.parametrize("mode", ["reference", "fp64", "mixed"])
@pytest.mark.parametrize("name,make", CG_CASES, ids=[c[0] for c in CG_CASES])
def test_flow_cg_matches_oracle(name, make, mode):
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = make()
    M.sort_indices()
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64)
    n = len(A) - 1
    rng = np.random.default_rng(n + 1)
    b, x0 = 1e3 * rng.uniform(-1.0, 1.0, n), 1e3 * rng.uniform(-1.0, 1.0, n)
    sysm = System(A, C, V)
    x = torch.from_numpy(x0).cuda()
    r = torch.zeros(n, dtype=torch.float64, device="cuda")
    # the reference rule is capped at N steps; the product modes get room beyond that
    info = sysm.solve(torch.from_numpy(b).cuda(), x, method="cg", mode=mode, precision=1e-12, residual=r,
                      max_iter=0 if mode == "reference" else 10 * n + 100)
    xh, rh = x.cpu().numpy(), r.cpu().numpy()
    K_o, x_o, _ = oracle.cg(A, C, V, b, x0=x0, precision=1e-12)
    assert info["status"] == (3 if mode == "reference" and K_o == n else 0), (info, K_o)
    assert np.linalg.norm(xh - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    assert np.linalg.norm(rh - (b - M @ xh)) <= 1e-6 * np.linalg.norm(b), info     # the drop-in's bar
    if mode == "reference":
        assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    else:
        assert np.linalg.norm(b - M @ xh) <= 1e-12 * np.linalg.norm(b), info
    # a capped solve stops after exactly that many steps, with x and r of that step
    if mode == "reference" and K_o > 6:
        x = torch.from_numpy(x0).cuda()
        info = sysm.solve(torch.from_numpy(b).cuda(), x, method="cg", mode=mode, precision=1e-12, max_iter=5, residual=r)
        xh, rh = x.cpu().numpy(), r.cpu().numpy()
        assert info["status"] == 3 and info["iterations"] == 5, info
        true = b - M @ xh
        assert np.linalg.norm(rh - true) <= 1e-12 * max(np.linalg.norm(b), np.linalg.norm(M @ x0)), info
    sysm.close()


@pytest.mark.parametrize("method,mode", [("rainbow", "reference"), ("rainbow", "fp64"), ("cg", "reference")])
def test_flow_solvers_repeat_bit_for_bit(method, mode):
    """Every sum is formed in a fixed order, whatever the order in which values arrive."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = _lattice(3, 2, 3, 0) if mode == "fp64" else _lattice(3, 1, 5, 0)
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data
    n = len(A) - 1
    sysm = System(A, C, V)
    sysm.set_rainbow(oracle.csr_diagonal(A, C, V), 1.0, *oracle.rainbow(A, C))
    b = torch.from_numpy(np.random.default_rng(1).uniform(-1e3, 1e3, n)).cuda()
    runs = []
    for _ in range(3):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        info = sysm.solve(b, x, method=method, mode=mode, precision=1e-10)
        runs.append((info["iterations"], x.cpu().numpy().tobytes()))
    assert runs[0] == runs[1] == runs[2]
    sysm.close()


SMALL_CASES = [("one_row", lambda: _diagonal(1)), ("diagonal", lambda: _diagonal(40)), ("tridiagonal_33", lambda: _tridiagonal(33)),
               ("arrow_257", lambda: _arrow(257)), ("p1_2d", lambda: _lattice(2, 1, 5, 1001)),
               ("p2_2d", lambda: _lattice(2, 2, 5, 0)), ("p1_3d_wide_levels", lambda: _lattice(3, 1, 5, 9000)),
               ("p2_3d_long_rows", lambda: _lattice(3, 2, 4, 9000)), ("p3_3d", lambda: _lattice(3, 3, 2, 0)),
               ("largest_colors", lambda: _lattice(2, 1, 7, 4608))]


@pytest.mark.parametrize("method,omega", [("ssor", 1.0), ("ssor", 1.4), ("rainbow", 1.0), ("rainbow", 0.8)])
@pytest.mark.parametrize("name,make", SMALL_CASES, ids=[c[0] for c in SMALL_CASES])
def test_one_block_solver_matches_oracle(name, make, method, omega):
    """One-block SSOR and multicolor PCG (kernels_small.cu): single rows, one and several lanes per
    row, phases wider than the staging slots, rows of several chunks, and rows with D == 0."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = make()
    M.sort_indices()
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64)
    n = len(A) - 1
    rng = np.random.default_rng(n + 2)
    b = 1e3 * rng.uniform(-1.0, 1.0, n)
    diag = oracle.csr_diagonal(A, C, V)
    sysm = System(A, C, V)
    if method == "ssor":
        sysm.set_ssor(diag, omega)
        K_o, x_o, _ = oracle.cg_ssor(A, C, V, b, diag, omega, precision=1e-11)
    else:
        rb = oracle.rainbow(A, C)
        sysm.set_rainbow(diag, omega, *rb)
        K_o, x_o, _ = oracle.cg_rainbow(A, C, V, b, diag, rb, omega, precision=1e-11)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = sysm.solve(torch.from_numpy(b).cuda(), x, method=method, mode="reference", precision=1e-11)
    assert info["status"] == (3 if K_o == n else 0), (info, K_o)
    assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    sysm.close()


@pytest.mark.parametrize("method", ["ssor", "rainbow"])
def test_one_block_solver_skips_zero_diagonal_rows(method):
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = _lattice(2, 1, 4, 0)
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data
    n = len(A) - 1
    b = np.random.default_rng(4).uniform(-1e3, 1e3, n)
    diag = oracle.csr_diagonal(A, C, V)
    diag[[3, 77, n - 1]] = 0.0
    sysm = System(A, C, V)
    if method == "ssor":
        sysm.set_ssor(diag, 1.0)
        K_o, x_o, _ = oracle.cg_ssor(A, C, V, b, diag, 1.0, precision=1e-11)
    else:
        rb = oracle.rainbow(A, C)
        sysm.set_rainbow(diag, 1.0, *rb)
        K_o, x_o, _ = oracle.cg_rainbow(A, C, V, b, diag, rb, 1.0, precision=1e-11)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = sysm.solve(torch.from_numpy(b).cuda(), x, method=method, mode="reference", precision=1e-11)
    assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    sysm.close()


MORE_CASES = CASES + [("scaled_identity", lambda: 2.0 * sp.identity(70, format="csr")),
                      ("tridiagonal_5000", lambda: _tridiagonal(5000)), ("p1_2d", lambda: _lattice(2, 1, 6, 0)),
                      ("many_rows_published", lambda: _lattice(3, 1, 5, 30_011)),
                      ("p2_published", lambda: _lattice(3, 2, 4, 0)),
                      ("empty_rows", lambda: _lattice(2, 1, 4, 0)),
                      ("rows_90011", lambda: _lattice(3, 1, 6, 90_011)),
                      ("rows_200017", lambda: _lattice(3, 1, 6, 200_017))]


@pytest.mark.parametrize("solver", ["minres", "cr"])
@pytest.mark.parametrize("name,make", MORE_CASES, ids=[c[0] for c in MORE_CASES])
def test_minres_and_cr_match_oracle(cuda, name, make, solver):
    """MINRES and conjugate residuals with one sum per iteration, vectors in registers and in
    memory; a matrix whose Lanczos vectors end at once (the expanded norm cancels); rows without
    entries (their b is 0). K within 2% (at least 1) of the oracle, the solution within 1e-9 of it."""
    import simplefem_gb300 as S
    from oracle import oracle
    M = make()
    n = M.shape[0]
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    if name == "empty_rows":
        keep = np.ones(n)
        keep[[0, 5, n - 1]] = 0.0
        M = (sp.diags(keep) @ M @ sp.diags(keep)).tocsr()
        M.eliminate_zeros()
        b *= keep
    M.sort_indices()
    A, C, V = M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64)
    x = np.zeros(n)
    res = np.full(n, np.nan)
    fn = S.MINRESCSR if solver == "minres" else S.ConjugateResidualSolverCSR
    K = fn(n, x, b, A, C, V, res, 1e-11, -3)
    info = S.last_info()
    K_o, x_o, _ = (oracle.minres if solver == "minres" else oracle.cr)(A, C, V, b, precision=1e-11)
    # the iteration cap is N: tiny systems may end on it with the exact solution
    assert info["status"] == 0 or (info["status"] == 3 and K == n and K_o >= n - 1), info
    assert abs(K - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (K, K_o)
    assert np.linalg.norm(x - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    # MINRES returns the true residual, CR its recursion's: both are at the solution's accuracy
    assert np.linalg.norm(res - (b - M @ x)) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [1, 31, 1025, 8191, 8193, 65_537, 300_001])
def test_norms_over_blocks(cuda, n):
    """The right-hand side's norm (one cluster of eight blocks, 8192 values a step) and the true
    residual's, through the reported quotient of the two, against numpy: a sum of n squares is off by at most a few units per addition in
    a chain, here n / 8192 + 30 of them, far below 1e-13."""
    import torch
    from simplefem_gb300.system import System
    M = _diagonal(n) if n < 3 else _tridiagonal(n)
    M.sort_indices()
    sysm = System(M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64))
    rng = np.random.default_rng(n)
    b, x0 = rng.uniform(-1.0, 1.0, n), rng.uniform(-1.0, 1.0, n)
    x = torch.from_numpy(x0).cuda()
    info = sysm.solve(torch.from_numpy(b).cuda(), x, method="cg", mode="fp64", precision=1e-3, max_iter=1)
    xh = x.cpu().numpy()
    rel = np.linalg.norm(b - M @ xh) / np.linalg.norm(b)
    assert abs(info["true_relres"] - rel) <= 1e-13 * max(rel, 1.0), (info, rel)
    sysm.close()


@pytest.mark.parametrize("scaling", [1.0, -0.75])
@pytest.mark.parametrize("length", [1, 4, 5, 6, 7, 8, 14, 15, 16, 64, 65, 66, 72, 73, 130])
def test_product_over_slice_lengths(cuda, length, scaling):
    """y = scaling A x for slices of one length each around the chunk lengths (5, 7, 8), a last slice
    that is not full and rows without entries among them. A row of k entries is off by at most k
    units of rounding of its sum of magnitudes, plus one for the scaling."""
    import torch
    from simplefem_gb300.system import System
    n = 32 * 5 + 9
    rng = np.random.default_rng(length)
    counts = np.full(n, length)
    counts[[3, 40]] = 0
    A = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    C = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in counts]).astype(np.int32)
    V = rng.standard_normal(len(C))
    x = rng.standard_normal(n)
    M = sp.csr_matrix((V, C, A), shape=(n, n))
    s = System(A, C, V)
    y = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    s.apply(torch.from_numpy(x).cuda(), y, scaling)
    y = y.cpu().numpy()
    bound = (length + 1) * np.finfo(np.float64).eps * abs(scaling) * (abs(M) @ np.abs(x))
    assert (np.abs(y - scaling * (M @ x)) <= bound).all()
    s.close()
