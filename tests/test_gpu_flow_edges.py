"""Edges of the dataflow and one-block solvers: blocks whose warps hold slices of different shapes,
solves that end at the iteration cap, the smallest systems, and set-up for uneven rows."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

pytestmark = pytest.mark.gpu


def _csr(M):
    M = M.tocsr()
    M.sort_indices()
    return M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data.astype(np.float64)


def _tridiagonal(n):
    return sp.diags([-np.ones(n - 1), np.full(n, 2.5), -np.ones(n - 1)], [-1, 0, 1]).tocsr()


def _long_and_short(long, short, per_row, seed=7):
    """`long` rows of about `per_row` entries coupled to a tridiagonal rest of `short` rows: symmetric
    and strictly diagonally dominant."""
    rng = np.random.default_rng(seed)
    k = long * (per_row - 1) // 2
    R = sp.coo_matrix((-rng.uniform(0.1, 1.0, k), (rng.integers(0, long, k), rng.integers(0, long, k))), shape=(long, long))
    R = R + R.T
    R.setdiag(0.0)
    M = sp.bmat([[R, None], [None, _tridiagonal(short)]]).tolil()
    M[long - 1, long] = M[long, long - 1] = -0.25
    M = M.tocsr()
    off = abs(M - sp.diags(M.diagonal()))
    return (M - sp.diags(M.diagonal()) + sp.diags(np.asarray(off.sum(axis=1)).ravel() * 1.02 + 0.1)).tocsr()


@pytest.mark.parametrize("mode", ["reference", "fp64", "mixed"])
@pytest.mark.parametrize("long,short,per_row", [(600, 3000, 40), (40, 500, 30), (1000, 33, 12), (64, 64, 60)])
def test_cg_blocks_with_slices_of_different_shapes(long, short, per_row, mode):
    """Plain CG with its vectors in registers, where the warps of a block hold rows of one, two and
    many lanes each or no rows at all. K within 2% (at least 1) of the oracle, the solution within
    1e-9 of it."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = _long_and_short(long, short, per_row)
    A, C, V = _csr(M)
    n = len(A) - 1
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    K_o, x_o, _ = oracle.cg(A, C, V, b, precision=1e-12)
    if mode != "reference" and K_o == n:      # the oracle's own cap is N
        x_o = sp.linalg.spsolve(M.tocsc(), b)
    s = System(A, C, V)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    # the reference rule is capped at N steps; the product modes get room beyond that
    info = s.solve(torch.from_numpy(b).cuda(), x, method="cg", mode=mode, precision=1e-12,
                   max_iter=0 if mode == "reference" else 10 * n + 100)
    assert info["status"] == (3 if mode == "reference" and K_o == n else 0), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    if mode == "reference":
        assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    s.close()


def _lattice(dim, r, L, n):
    from simplefem_gb300 import workloads
    A, C, V = workloads.lattice_matrix(dim, r, L, 3)
    M = sp.csr_matrix((V, C, A))
    return M[:n, :n].tocsr() if n else M


# (operator, cap): the cap that the drop-ins default to (N) on systems that are exact there, and
# one in the middle of a solve in each form of the kernels
CAPPED = [("one_row", lambda: sp.csr_matrix([[3.7]]), 1), ("two_rows", lambda: _tridiagonal(2), 2),
          ("identity_row", lambda: 0.3 * sp.identity(50, format="csr"), 1), ("three_rows", lambda: _tridiagonal(3), 3),
          ("registers", lambda: _lattice(2, 1, 5, 0), 9), ("published", lambda: _lattice(3, 2, 4, 20_011), 5),
          ("barrier", lambda: _lattice(3, 1, 6, 81_001), 5)]


@pytest.mark.parametrize("method", ["cg", "rainbow_eisenstat", "rainbow"])
@pytest.mark.parametrize("name,make,cap", CAPPED, ids=[c[0] for c in CAPPED])
def test_capped_solve_reports_the_norm_of_its_residual(name, make, cap, method):
    """final_norm of a solve that ends at the cap is the norm of the residual it returns: ||r|| for
    plain CG, sqrt(z.r) with z = S r for Eisenstat's form, whose r is the one S scales (omega = 1:
    S = D). A sum of n squares is off by at most a few units per addition in a chain, of which there
    are far fewer than 1000 here: 1e-12. For the two-sweep form, whose z is not returned: that the
    reported z.r is no more than that of an exact solve's rounding on the exact systems."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = make()
    A, C, V = _csr(M)
    n = len(A) - 1
    diag = oracle.csr_diagonal(A, C, V)
    s = System(A, C, V)
    if method != "cg":
        s.set_rainbow(diag, 1.0, *oracle.rainbow(A, C))
    for seed in range(12 if n < 100 else 1):
        b = 1e3 * np.random.default_rng(seed).uniform(-1.0, 1.0, n)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        r = torch.zeros(n, dtype=torch.float64, device="cuda")
        info = s.solve(torch.from_numpy(b).cuda(), x, method=method, mode="reference", precision=1e-300, max_iter=cap,
                       residual=r)
        if info["status"] == 0:      # below the drop-ins' absolute floor already
            continue
        assert info["status"] == 3 and info["iterations"] == cap, info
        rh = r.cpu().numpy()
        if method == "cg":
            norm = np.linalg.norm(rh)
        elif method == "rainbow_eisenstat":
            norm = np.sqrt(np.sum(diag * rh * rh))
        else:
            if cap >= n:
                assert info["final_norm"] <= 1e-12 * np.sqrt(np.sum(b * b / diag)), info
            continue
        assert abs(info["final_norm"] - norm) <= 1e-12 * norm, (info, norm)
    s.close()


@pytest.mark.parametrize("n", [700, 200_003])
def test_a_dense_row_is_set_up_in_linear_time(n):
    """A dense first row and column: parts of more entries than are ordered at once. The first solve
    of 200,003 rows, slices included, stays below a second and a half (its entries compared pair by
    pair take several); the solution within 1e-9 of the oracle's and K within 2% (at least 1)."""
    import time
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    rest = np.arange(1, n)
    rows = np.concatenate([np.zeros(n, int), rest, rest])
    cols = np.concatenate([np.arange(n), np.zeros(n - 1, int), rest])
    vals = np.concatenate([[3.0], np.full(n - 1, 0.5 / n), np.full(n - 1, 0.5 / n), np.linspace(1.0, 2.0, n - 1)])
    M = sp.csr_matrix((vals, (rows, cols)), shape=(n, n))
    A, C, V = _csr(M)
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    diag = oracle.csr_diagonal(A, C, V)
    rb = oracle.rainbow(A, C)
    K_o, x_o, _ = oracle.cg_rainbow(A, C, V, b, diag, rb, 1.0, precision=1e-11)
    s = System(A, C, V)
    s.set_rainbow(diag, 1.0, *rb)
    bd, x = torch.from_numpy(b).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    t = time.perf_counter()
    info = s.solve(bd, x, method="rainbow_eisenstat", mode="reference", precision=1e-11)
    torch.cuda.synchronize()
    t = time.perf_counter() - t
    assert info["status"] == 0 and abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    assert t < 1.5, t
    s.close()


@pytest.mark.parametrize("method", ["ssor", "rainbow"])
def test_memory_counts_the_one_block_solvers_tables(method):
    """The first solve of a small system lays out full rows (12 bytes an entry) and staged sweep
    slices: memory_bytes grows by at least the former."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    A, C, V = _csr(_lattice(2, 1, 6, 0))
    n = len(A) - 1
    diag = oracle.csr_diagonal(A, C, V)
    s = System(A, C, V)
    if method == "ssor":
        s.set_ssor(diag, 1.0)
    else:
        s.set_rainbow(diag, 1.0, *oracle.rainbow(A, C))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    b = torch.ones_like(x)
    s.solve(b, x, method="cg", mode="reference", precision=1e-6)      # the work vectors
    before = s.memory_bytes()
    s.solve(b, x, method=method, mode="reference", precision=1e-6)
    assert s.memory_bytes() >= before + 12 * len(C)
    s.close()


def _chain_and_rows(chain, rows):
    """Levels of one row each (a chain) beside one level of many rows."""
    return sp.block_diag([_tridiagonal(chain), sp.diags(np.linspace(1.0, 2.0, rows))]).tocsr()


LEVELS = [("chain_3000_and_1500", lambda: _chain_and_rows(3000, 1500)), ("chain_8000_and_600", lambda: _chain_and_rows(8000, 600)),
          ("chain_9001", lambda: _chain_and_rows(9000, 1)), ("p1_2d_12700", lambda: _lattice(2, 1, 7, 12_700)),
          ("p1_2d_last_in_one_block", lambda: _lattice(2, 1, 7, 13_569)), ("p1_2d_first_beyond", lambda: _lattice(2, 1, 7, 13_570)),
          ("p2_3d_13500", lambda: _lattice(3, 2, 4, 13_500)), ("p1_3d_13000", lambda: _lattice(3, 1, 5, 13_000))]


@pytest.mark.parametrize("name,make", LEVELS, ids=[c[0] for c in LEVELS])
def test_index_order_schedules_of_uneven_levels(name, make):
    """Index-order SSOR where the staged slots cannot hold the widest level: a wide level among
    levels of one row, and systems up to the last that fits a block (vectors that leave room for two
    slices a slot). K within 2% (at least 1) of the oracle, the solution within 1e-9 of it; the
    tables stay a small multiple of the matrix: a slot's slices hold 32 rows in 1,360 bytes, at most
    four are staged for one that holds rows, over two sweeps, beside 12 bytes per entry, columns of
    32 of them padded to the longest of 32 rows (six times the entries here at most)."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = make()
    A, C, V = _csr(M)
    n = len(A) - 1
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    diag = oracle.csr_diagonal(A, C, V)
    K_o, x_o, _ = oracle.cg_ssor(A, C, V, b, diag, 1.0, precision=1e-10)
    s = System(A, C, V)
    s.set_ssor(diag, 1.0)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    bd = torch.from_numpy(b).cuda()
    s.solve(bd, x, method="cg", mode="reference", precision=1e-2)
    before = s.memory_bytes()
    x.zero_()
    info = s.solve(bd, x, method="ssor", mode="reference", precision=1e-10)
    assert info["status"] == 0, info
    assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    if name.startswith("chain"):
        assert s.memory_bytes() - before <= 2 * 4 * 1360 * (n // 32 + n) + 6 * 12 * len(C)
    s.close()


@pytest.mark.parametrize("method,mode", [("rainbow", "fp64"), ("rainbow", "mixed"), ("rainbow_eisenstat", "reference"),
                                         ("cg", "fp64")])
def test_small_solves_on_several_streams_share_the_gpu(method, mode):
    """Eight threads with a stream and a system of 4,225 rows each: the results are those of a solve
    alone, bit for bit, and together they take less than half of the time of one after the other
    (they fit the SMs side by side)."""
    import threading
    import time
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    A, C, V = _csr(_lattice(2, 1, 6, 0))
    n = len(A) - 1
    diag, rb = oracle.csr_diagonal(A, C, V), oracle.rainbow(A, C)
    T, reps = 8, 6
    b = torch.from_numpy(1e3 * np.random.default_rng(3).uniform(-1.0, 1.0, n)).cuda()
    systems, xs = [], []
    for _ in range(T):
        s = System(A, C, V)
        s.set_rainbow(diag, 1.0, *rb)
        systems.append(s)
        xs.append(torch.zeros_like(b))
    streams = [torch.cuda.Stream() for _ in range(T)]

    def solve(i):
        with torch.cuda.stream(streams[i]):
            xs[i].zero_()
            systems[i].solve(b, xs[i], method=method, mode=mode, precision=1e-10)

    torch.cuda.synchronize()
    for _ in range(3):          # layouts and, for mixed, the choice of the inner precision
        for i in range(T):
            solve(i)
    alone = [x.cpu().numpy().tobytes() for x in xs]
    t = time.perf_counter()
    for _ in range(reps):
        for i in range(T):
            solve(i)
    torch.cuda.synchronize()
    serial = time.perf_counter() - t
    gate = threading.Barrier(T + 1)

    def worker(i):
        gate.wait()
        for _ in range(reps):
            solve(i)
        gate.wait()

    together = []
    for _ in range(3):          # the best counts: the host may be interrupted
        threads = [threading.Thread(target=worker, args=(i,)) for i in range(T)]
        for th in threads:
            th.start()
        gate.wait()
        t = time.perf_counter()
        gate.wait()
        together.append(time.perf_counter() - t)
        for th in threads:
            th.join()
        torch.cuda.synchronize()
        assert [x.cpu().numpy().tobytes() for x in xs] == alone
    assert min(together) < 0.5 * serial, (together, serial)
    for s in systems:
        s.close()


@pytest.mark.parametrize("length", [8, 16, 40, 64, 72])
def test_product_reads_no_entry_that_a_row_does_not_have(cuda, length):
    """Rows of whole chunks of eight entries that do not touch unknown 0 are finite when x is infinite
    there. A row of k entries is off by at most k units of rounding of its sum of magnitudes."""
    import torch
    from simplefem_gb300.system import System
    n = 32 * 6 + 5
    rng = np.random.default_rng(length)
    A = (np.arange(n + 1) * length).astype(np.int32)
    C = np.concatenate([np.sort(1 + rng.choice(n - 1, length, replace=False)) for _ in range(n)]).astype(np.int32)
    V = rng.standard_normal(len(C))
    x = rng.standard_normal(n)
    M = sp.csr_matrix((V, C, A), shape=(n, n))
    exact, bound = M @ x, length * np.finfo(np.float64).eps * (abs(M) @ np.abs(x))
    x[0] = np.inf
    s = System(A, C, V)
    y = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    s.apply(torch.from_numpy(x).cuda(), y)
    assert (np.abs(y.cpu().numpy() - exact) <= bound).all()
    s.close()


@pytest.mark.parametrize("n", [1, 31, 255, 257, 511, 513, 1023, 1025, 2047, 2049, 4096, 6145])
@pytest.mark.parametrize("method", ["cg", "rainbow_eisenstat"])
def test_slices_at_the_edges_of_their_windows(n, method):
    """Rows are cut in windows of 256 rows of a color and 512 of a matrix, which is sorted in windows of
    2,048: counts around them, rows without entries beside the diagonal, and one row far longer than the rest in the
    last window. K within 2% (at least 1) of the oracle, the solution within 1e-9 of it."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    rng = np.random.default_rng(n)
    M = sp.diags(rng.uniform(3.0, 4.0, n)).tolil()
    for i in rng.integers(0, n, n):
        j = int(rng.integers(max(0, i - 40), i + 1))
        if i != j:
            M[i, j] = M[j, i] = -0.1
    if n > 1000:
        for j in range(n - 900, n - 1, 3):
            M[n - 1, j] = M[j, n - 1] = -0.002
    A, C, V = _csr(M)
    b = 1e3 * rng.uniform(-1.0, 1.0, n)
    diag, rb = oracle.csr_diagonal(A, C, V), oracle.rainbow(A, C)
    s = System(A, C, V)
    if method == "cg":
        K_o, x_o, _ = oracle.cg(A, C, V, b, precision=1e-11)
    else:
        K_o, x_o, _ = oracle.cg_rainbow(A, C, V, b, diag, rb, 1.0, precision=1e-11)
        s.set_rainbow(diag, 1.0, *rb)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = s.solve(torch.from_numpy(b).cuda(), x, method=method, mode="reference", precision=1e-11)
    assert info["status"] == (3 if K_o == n else 0), (info, K_o)
    assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    s.close()


@pytest.mark.parametrize("method", ["cg", "rainbow"])
def test_slices_cost_no_more_than_a_few_iterations(method):
    """The first solve of 274,625 rows, slices included, takes at most 2 ms more than the second
    (cut on the device 0.3 ms; 2.6 ms for plain CG and 6.7 for the colors when a host walk cut them).
    The best of three systems counts."""
    import time
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    A, C, V = _csr(_lattice(3, 1, 6, 0) + 30.0 * sp.identity(65 ** 3))
    n = len(A) - 1
    diag, rb = oracle.csr_diagonal(A, C, V), oracle.rainbow(A, C)
    b = torch.from_numpy(1e3 * np.random.default_rng(0).uniform(-1.0, 1.0, n)).cuda()
    extra = []
    for _ in range(4):          # the first fills the memory pool
        s = System(A, C, V)
        if method == "rainbow":
            s.set_rainbow(diag, 1.0, *rb)
        times = []
        for _ in range(3):
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            t = time.perf_counter()
            info = s.solve(b, x, method=method, mode="fp64", precision=1e-6)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
            assert info["status"] == 0, info
        extra.append(times[0] - min(times[1:]))
        s.close()
    assert min(extra[1:]) < 2e-3, extra


@pytest.mark.parametrize("n,width", [(700, 399), (700, 401), (500, 500)])
def test_residual_of_long_rows(n, width):
    """The true residual of rows on either side of 400 entries on average, through the reported
    quotient with the right-hand side's norm, against numpy: sums of `width` products and of n squares
    are off by a few hundred units at most, 1e-12."""
    import torch
    from simplefem_gb300.system import System
    rng = np.random.default_rng(width)
    M = np.zeros((n, n))
    for i in range(n):
        M[i, (i + np.arange(width)) % n] = rng.uniform(-1.0, 1.0, width)
    M += np.diag(np.full(n, 2.0 * width))
    A, C, V = _csr(sp.csr_matrix(M))
    s = System(A, C, V)
    b, x0 = rng.uniform(-1.0, 1.0, n), rng.uniform(-1.0, 1.0, n)
    x = torch.from_numpy(x0).cuda()
    info = s.solve(torch.from_numpy(b).cuda(), x, method="cg", mode="fp64", precision=1e-3, max_iter=1)
    rel = np.linalg.norm(b - M @ x.cpu().numpy()) / np.linalg.norm(b)
    assert abs(info["true_relres"] - rel) <= 1e-12 * max(rel, 1.0), (info, rel)
    s.close()


@pytest.mark.parametrize("kind,site", [(1, 78), (2, 0)], ids=["published_value", "staged_copy"])
def test_waits_for_values_and_copies_give_up(cuda, kind, site):
    """A wait that nothing satisfies ends after the solvers' limit (4 s) with FEEC_TIMEOUT and its site, and
    the GPU goes on working: a solve right after gives the solution to 1e-9."""
    import ctypes
    import torch
    from simplefem_gb300 import _native
    from simplefem_gb300.system import System
    lib = _native.gpu()
    st, at, ms = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_double(0.0)
    assert lib.feec_selftest_solver_wait(kind, ctypes.byref(st), ctypes.byref(at), ctypes.byref(ms)) == _native.FEEC_OK
    assert st.value == 4 and at.value == site
    assert 4000.0 <= ms.value < 9000.0, ms.value
    for bad in (-1, 0, 3):
        assert lib.feec_selftest_solver_wait(bad, ctypes.byref(st), ctypes.byref(at), ctypes.byref(ms)) == 6
    A, C, V = _csr(_tridiagonal(1000))
    s = System(A, C, V)
    x = torch.zeros(1000, dtype=torch.float64, device="cuda")
    b = np.random.default_rng(0).uniform(-1.0, 1.0, 1000)
    s.solve(torch.from_numpy(b).cuda(), x, method="cg", mode="fp64", precision=1e-11)
    x_o = sp.linalg.spsolve(_tridiagonal(1000).tocsc(), b)
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o)
    s.close()


@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("method,mode", [("rainbow", "reference"), ("rainbow_eisenstat", "reference"), ("rainbow", "fp64"),
                                         ("rainbow", "mixed"), ("cg", "reference"), ("cg", "mixed")])
def test_one_and_two_rows_converge_beyond_the_cap(method, mode, n):
    """The smallest systems, with room for the step after which they are exact: one slice, one block.
    The solution within 1e-12 (cond < 3, residual below 1e-13 of b)."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    M = _tridiagonal(n)
    A, C, V = _csr(M)
    s = System(A, C, V)
    s.set_rainbow(oracle.csr_diagonal(A, C, V), 1.0, *oracle.rainbow(A, C))
    for seed in range(8):
        b = 1e3 * np.random.default_rng(seed).uniform(-1.0, 1.0, n)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        info = s.solve(torch.from_numpy(b).cuda(), x, method=method, mode=mode, precision=1e-13, max_iter=20)
        exact = np.linalg.solve(M.toarray(), b)
        assert info["status"] == 0 and info["iterations"] <= 20, info
        assert np.linalg.norm(x.cpu().numpy() - exact) <= 1e-12 * np.linalg.norm(exact), info
    s.close()


def test_small_solves_of_different_sizes_on_threads():
    """The one-block solver's shared memory differs by system, its kernel's limit does not: threads
    that solve small and large systems at the same time, 3,000 capped solves each, all launch."""
    import threading
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    failed = []

    def worker(n, gate):
        A, C, V = _csr(_lattice(2, 1, 7, n))
        s = System(A, C, V)
        s.set_ssor(oracle.csr_diagonal(A, C, V), 1.0)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            b = torch.ones(n, dtype=torch.float64, device="cuda")
            x = torch.zeros_like(b)
            gate.wait()
            for _ in range(3000):
                try:
                    s.solve(b, x, method="ssor", mode="reference", precision=1e-12, max_iter=1)
                except Exception as e:      # reported by the test's own thread
                    failed.append((n, repr(e)))
                    break
        s.close()

    sizes = (60, 100, 60, 13_000, 13_000, 13_000, 60, 13_500)
    gate = threading.Barrier(len(sizes))
    threads = [threading.Thread(target=worker, args=(n, gate)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("dim,r,L,count", [(2, 1, 6, 100), (2, 1, 6, 200), (3, 2, 3, 64), (3, 2, 3, 200), (3, 1, 4, 100)])
def test_teams_of_a_batch_pay(dim, r, L, count):
    """Equal systems that do not fit the GPU in teams of several blocks, or whose colors are too short
    for them: the batch takes at most 1.15 times as long as with one block per system (up to twice as
    long before teams were weighed against them), and the solutions agree to 1e-9."""
    import torch
    from oracle import oracle
    from simplefem_gb300 import system
    A, C, V = _csr(_lattice(dim, r, L, 0))
    n = len(A) - 1
    s = system.System(A, C, V)
    s.set_rainbow(oracle.csr_diagonal(A, C, V), 1.0, *oracle.rainbow(A, C))
    g = torch.Generator(device="cuda")
    g.manual_seed(count)
    bs = list((torch.rand(count, n, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0).unbind())
    times, results = [], []
    for threads in (256, 0):
        xs = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(count)]
        batch = system.Batch([s] * count, bs, xs, method="rainbow", mode="fp64", precision=1e-10, team_threads=threads)
        ms = []
        for _ in range(4):
            for x in xs:
                x.zero_()
            infos, t = batch.run()
            ms.append(t)
        assert all(i["status"] == 0 for i in infos)
        times.append(min(ms))
        results.append(torch.stack(xs))
        batch.close()
    s.close()
    assert times[1] <= 1.15 * times[0], times
    assert torch.linalg.norm(results[0] - results[1]) <= 1e-9 * torch.linalg.norm(results[0])


@pytest.mark.parametrize("solver", ["minres", "cr"])
@pytest.mark.parametrize("n,half", [(5600, 124), (5600, 126), (11_300, 62), (11_300, 65)])
def test_minres_and_cr_of_long_rows(cuda, n, half, solver):
    """Banded rows on either side of the line between the two forms (128 entries a row, 1.4 M entries): K
    within 2% (at least 1) of the oracle, the solution within 1e-9 of it."""
    import simplefem_gb300 as S
    from oracle import oracle
    off = np.arange(1, half + 1)
    R = sp.diags([-np.ones(n - o) for o in off], off, shape=(n, n))
    R = (R + R.T).tocsr()
    A, C, V = _csr(R + sp.diags(np.asarray(abs(R).sum(axis=1)).ravel() * 1.01 + 1.0))
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    x, res = np.zeros(n), np.zeros(n)
    K = (S.MINRESCSR if solver == "minres" else S.ConjugateResidualSolverCSR)(n, x, b, A, C, V, res, 1e-11, -3)
    K_o, x_o, _ = (oracle.minres if solver == "minres" else oracle.cr)(A, C, V, b, precision=1e-11)
    assert abs(K - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (K, K_o)
    assert np.linalg.norm(x - x_o) <= 1e-9 * np.linalg.norm(x_o)


@pytest.mark.parametrize("mode", ["reference", "mixed"])
@pytest.mark.parametrize("half", [196, 204])
def test_cg_of_many_long_rows(half, mode):
    """Plain CG on 20,000 banded rows on either side of 8 M stored entries, beyond which d is not
    published. K within 2% (at least 1) of the oracle, the solution within 1e-9 of it."""
    import torch
    from oracle import oracle
    from simplefem_gb300.system import System
    n = 20_000
    off = np.arange(1, half + 1)
    R = sp.diags([-np.ones(n - o) for o in off], off, shape=(n, n))
    R = (R + R.T).tocsr()
    A, C, V = _csr(R + sp.diags(np.asarray(abs(R).sum(axis=1)).ravel() * 1.01 + 1.0))
    b = 1e3 * np.random.default_rng(n).uniform(-1.0, 1.0, n)
    K_o, x_o, _ = oracle.cg(A, C, V, b, precision=1e-12)
    s = System(A, C, V)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = s.solve(torch.from_numpy(b).cuda(), x, method="cg", mode=mode, precision=1e-12)
    assert info["status"] == 0, info
    assert np.linalg.norm(x.cpu().numpy() - x_o) <= 1e-9 * np.linalg.norm(x_o), info
    if mode == "reference":
        assert abs(info["iterations"] - K_o) <= max(1, int(np.ceil(0.02 * K_o))), (info, K_o)
    s.close()
