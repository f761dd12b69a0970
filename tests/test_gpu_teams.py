"""The kernels a batch of systems or of right-hand sides is sent to by its size. Batches whose systems differ so much that the large ones are solved by clusters of blocks: every
system reaches 1e-10 with the exact solution to 1e-9 (the bounds of the batched engine's other
tests), and agrees with one-block teams, for every cluster size and in both entry points."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

pytestmark = pytest.mark.gpu

# (polynomial degree, refinement) of 2D systems; P1 has (2^L + 1)^2 rows
MIXES = {
    "one_large": [(1, 8)],                                         # 16 blocks
    "every_size": [(1, 8), (1, 7), (2, 6), (1, 6), (2, 4), (1, 4), (1, 1)],
    "below_a_cluster": [(1, 5)] * 3,                               # 1,089 rows: one block each
    "many_small_one_large": [(1, 3)] * 40 + [(2, 6)],
    "more_teams_than_fit": [(1, 6)] * 200 + [(1, 7)] * 9,
}


def _system(degree, level, seed, method, dim=2):
    import simplefem_gb300 as S
    from simplefem_gb300 import workloads
    from simplefem_gb300.system import System
    A, C, V = workloads.lattice_matrix(dim, degree, level, seed)
    n = len(A) - 1
    s = System(A, C, V)
    if method == "rainbow":
        mat = S.MatrixCSR(n, n, A, C, V)
        rb = S.Rainbow(mat)
        s.set_rainbow(mat.getDiagonal().raw(), 1.0, rb.num_colors, rb.F, rb.B, rb.R)
    return s, sp.csr_matrix((V, C, A), shape=(n, n))


@pytest.mark.parametrize("method,mode", [("rainbow", "fp64"), ("rainbow", "mixed"), ("cg", "fp64"), ("cg", "mixed")])
@pytest.mark.parametrize("mix", sorted(MIXES))
def test_teams_by_system_size(cuda, mix, method, mode):
    torch = cuda
    from simplefem_gb300 import workloads
    from simplefem_gb300.system import Batch, solve_many
    made = {}
    systems, mats = [], []
    for (r, L) in MIXES[mix]:
        if (r, L) not in made:
            made[r, L] = _system(r, L, 10 * L + r, method)
        systems.append(made[r, L][0])
        mats.append(made[r, L][1])
    hb = [workloads.uniform_vector(900 + i, s.n) for i, s in enumerate(systems)]
    bs = [torch.from_numpy(b).cuda() for b in hb]

    def zeros():
        return [torch.zeros(s.n, dtype=torch.float64, device="cuda") for s in systems]

    xs, ys, zs = zeros(), zeros(), zeros()
    batch = Batch(systems, bs, xs, method=method, mode=mode, precision=1e-10)
    infos, _ = batch.run()
    batch.close()
    blocks = infos[0]["grid_blocks"]
    if mix in ("one_large", "every_size", "many_small_one_large"):
        assert blocks > len(systems)
    elif mix == "below_a_cluster":
        assert blocks == len(systems)
    once = solve_many(systems, bs, ys, method=method, mode=mode, precision=1e-10)
    one = Batch(systems, bs, zs, method=method, mode=mode, precision=1e-10, team_threads=256)
    plain, _ = one.run()
    one.close()
    assert plain[0]["grid_blocks"] <= len(systems)
    lu = {k: sla.splu(m.tocsc()) for k, (_, m) in made.items()}
    for i, (s, M) in enumerate(zip(systems, mats)):
        b = hb[i]
        exact = lu[MIXES[mix][i]].solve(b)
        for info, x in ((infos[i], xs[i]), (once[i], ys[i]), (plain[i], zs[i])):
            x = x.cpu().numpy()
            assert info["status"] == 0, (i, info)
            assert np.linalg.norm(b - M @ x) <= 1e-10 * np.linalg.norm(b)
            assert np.linalg.norm(x - exact) <= 1e-9 * np.linalg.norm(exact)
    for s, _ in made.values():
        s.close()


@pytest.mark.parametrize("method", ["rainbow", "cg"])
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("dim,degree,level", [(2, 1, 3), (2, 2, 4), (3, 1, 3), (3, 2, 2)])
def test_half_filled_launch_of_columns(cuda, dim, degree, level, threads, method):
    """Four columns per team: launches whose teams fill at most half of the SMs' threads take the
    kernel with long chunks of entries, fuller ones the other; rows of 3 to 60 entries give blocks
    below, at and above both chunk lengths. Every column meets 1e-10 and the exact solution to 1e-9
    (the bounds of the batched engine's other tests), a last team with one column included."""
    torch = cuda
    from simplefem_gb300 import workloads
    s, M = _system(degree, level, 7, method, dim)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 4 * sms * (512 // threads)            # the columns of the largest half-filled launch
    Bh = np.stack([workloads.uniform_vector(40 + j, s.n) for j in range(most + 1)])
    exact = sla.splu(M.tocsc()).solve(Bh.T).T
    s.set_batch_config(method, "mixed", 4, threads, 1)
    for columns in (1, 5, most, most + 1):
        B = torch.from_numpy(Bh[:columns].copy()).cuda()
        X = torch.zeros_like(B)
        # restarted CG may take more than the default budget of n iterations on 81 rows
        infos = s.solve_batch(B, X, method=method, mode="mixed", precision=1e-10, max_iter=20 * s.n)
        X = X.cpu().numpy()
        assert all(q["status"] == 0 for q in infos)
        res = np.linalg.norm(Bh[:columns] - (M @ X.T).T, axis=1)
        assert (res <= 1e-10 * np.linalg.norm(Bh[:columns], axis=1)).all()
        err = np.linalg.norm(X - exact[:columns], axis=1)
        assert (err <= 1e-9 * np.linalg.norm(exact[:columns], axis=1)).all()
    s.close()
