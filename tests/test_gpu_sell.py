"""GPU tests of the cycle's sliced operators (sell.cu), through the AMG solve
that uses them: fp64 solves take the oracle's iterations with x within 1e-9
of its (the bars of the block path, test_gpu_amg.py), on shapes that reach
each form: 16-bit offsets, 32-bit columns (a slice's columns spread over more
than 65,535), several lanes per row, ragged sizes, one long row, operators
that get no copy because long rows would pad their slices or one warp would
walk too long a slice, and reduced-precision storage."""
import numpy as np
import pytest
import torch

from gpu_util import AllocLog, sliced_steps, to_dev

pytestmark = pytest.mark.gpu


def _problem(orc, kind):
    if kind == "idx32":  # planes of 93,000 unknowns: a slice's columns span two of them
        return orc.laplacian(310, 300, 3), orc.geometric_hierarchy(310, 300, 3)
    if kind == "ragged":
        return orc.laplacian(61, 53, 47), orc.geometric_hierarchy(61, 53, 47)
    if kind == "lanes8":  # 24,360 rows of about 24 entries: eight lanes a row
        return orc.varcoef27(30, 29, 28, seed=4), orc.geometric_hierarchy(30, 29, 28)
    # "long_row_k": unknown k coupled to every other one (55,296 entries in row
    # k of its block row: more than 15 bits in either half of a packed count)
    import scipy.sparse as sp

    dims, k = (48, 48, 24), int(kind[-1])
    S = orc.laplacian(*dims).to_scipy().tolil()
    n = S.shape[0]
    others = np.arange(n) != k
    S[k, others] = -1e-4
    S[others, k] = -1e-4
    S = sp.csr_matrix(S)
    S = S + sp.diags(np.where(others, 1e-4, 1e-4 * n))
    S = sp.csr_matrix(S)
    S.sort_indices()
    return (orc.CSR(n, n, S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data),
            orc.geometric_hierarchy(*dims))


def _solver(A, Ps, **kw):
    from amgt_b200.amg import AmgSolver, default_params

    return AmgSolver(to_dev(A), [to_dev(P) for P in Ps], default_params(**kw))


@pytest.mark.parametrize("kind", ["idx32", "ragged", "lanes8", "long_row_0", "long_row_1", "long_row_3"])
def test_fp64_solve_matches_the_oracle(amgt, orc, kind):
    A, Ps = _problem(orc, kind)
    b = A.to_scipy() @ orc.rand_uniform(3, A.n)
    xo, it_o, _, _ = orc.Amg(A, Ps).solve(b)
    amgt.set_level_policy([0])
    try:
        with AllocLog(amgt) as log:
            S = _solver(A, Ps)
            x, it, rel = S.solve(torch.from_numpy(b).cuda())
            S.free()
    finally:
        amgt.set_level_policy([])
    assert (4 if kind == "idx32" else 2) * 32 * sliced_steps(A) in log.sizes  # level 0 is copied
    assert it == it_o and rel <= 1e-8
    assert np.linalg.norm(x.cpu().numpy() - xo) <= 1e-9 * np.linalg.norm(xo)


@pytest.mark.parametrize("prec", [1, 2, 3])
def test_reduced_levels_and_transfers_converge_fp64_verified(amgt, orc, prec):
    """Level 0's smoother at fp32, the coarser levels and the transfers at
    `prec` (fp32 / fp16 / bf16), on an operator no narrow storage holds
    exactly: the fp64 residual reaches 1e-8."""
    dims = (60, 58, 56)
    A, Ps = orc.varcoef27(*dims, seed=5), orc.geometric_hierarchy(*dims)
    b = A.to_scipy() @ orc.rand_uniform(4, A.n)
    amgt.set_level_policy([0, prec])
    try:
        with AllocLog(amgt) as log:
            S = _solver(A, Ps, flexible=1, smooth_prec0=1)
            x, it, rel = S.solve(torch.from_numpy(b).cuda())
            S.free()
    finally:
        amgt.set_level_policy([])
    steps = sliced_steps(A)  # level 0's copy: columns, 8-byte and 4-byte values
    assert all(k * 32 * steps in log.sizes for k in (2, 8, 4))
    r = b - A.to_scipy() @ x.cpu().numpy()
    assert np.linalg.norm(r) <= 1.0000001e-8 * np.linalg.norm(b)
    assert it < 60


def _coupled(orc, dims, rows, reach, count, seed=9):
    """7-point operator with `count` random couplings of each of `rows` to
    unknowns at most `reach` away (symmetric, diagonally dominant)."""
    import scipy.sparse as sp

    S = orc.laplacian(*dims).to_scipy()
    n, rng = S.shape[0], np.random.default_rng(seed)
    r = np.repeat(rows, count)
    c = np.concatenate([max(0, min(k - reach, n - 2 * reach - 1)) + rng.choice(2 * reach, count, replace=False)
                        for k in rows])
    E = sp.csr_matrix((np.full(r.size, 1e-3), (r, c)), shape=(n, n))
    E = E + E.T
    E.setdiag(0)
    S = sp.csr_matrix(S - E + sp.diags(np.asarray(E.sum(1)).ravel()))
    S.sort_indices()
    return orc.CSR(n, n, S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data)


@pytest.mark.parametrize("kind", ["padding", "one_slice", "full_blocks"])
def test_operators_that_get_no_copy(amgt, orc, kind):
    """One row of 60 entries in every slice (padded to seven times the
    entries), one slice of 1,000 steps in an operator of 75 MB, or full 4x4
    blocks (4 unknowns a node): no slice columns are allocated for level 0,
    and the solve converges as the block path does (fp64 residual)."""
    import scipy.sparse as sp

    from amgt_b200.amg import AmgSolver, default_params

    dims = {"padding": (61, 53, 47), "one_slice": (128, 128, 64), "full_blocks": (30, 29, 28)}[kind]
    n = int(np.prod(dims))
    Ps = orc.geometric_hierarchy(*dims)
    if kind == "full_blocks":
        def kron(M, B):
            K = sp.kron(M.to_scipy(), B).tocsr()
            K.sort_indices()
            return orc.CSR(K.shape[0], K.shape[1], K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data)

        A = kron(orc.laplacian(*dims), np.eye(4) + 0.1)
        Ps = [kron(P, np.eye(4)) for P in Ps]
    else:
        rows = np.arange(5, n, 32) if kind == "padding" else np.array([n // 2])
        A = _coupled(orc, dims, rows, 3000, 60 if kind == "padding" else 1000)
    assert orc.csr2bsr(A).nblk >= 65536
    b = A.to_scipy() @ orc.rand_uniform(6, A.n)
    steps = sliced_steps(A)
    assert (32 * steps > 2 * A.ja.size + 65536) == (kind == "padding")
    for M, copied in ((A, False), (orc.laplacian(*dims), True)):
        if copied and kind == "full_blocks":
            break
        amgt.set_level_policy([0])
        try:
            with AllocLog(amgt) as log:
                S = AmgSolver(to_dev(M), [to_dev(P) for P in Ps], default_params(exact_storage=0))
                if not copied:
                    x, it, rel = S.solve(torch.from_numpy(b).cuda())
                S.free()
        finally:
            amgt.set_level_policy([])
        assert log.sizes.count(2 * 32 * sliced_steps(M)) == int(copied)
    assert np.linalg.norm(b - A.to_scipy() @ x.cpu().numpy()) <= 1.0000001e-8 * np.linalg.norm(b)


def _solve_all(amgt, A, Ps, b, fail=None, multi=False):
    """Setup, solve (and a solve of two right-hand sides, and another solve)
    under the logging allocator."""
    amgt.set_level_policy([0])
    try:
        with AllocLog(amgt, fail) as log:
            S = _solver(A, Ps, exact_storage=0)
            out = [S.solve(b)]
            if multi:
                X, its, rel = S.solve_multi(torch.stack([b, b], 1).contiguous())
                out += [(X[:, 1].contiguous(), its[1], rel[1]), S.solve(b)]
            S.free()
    finally:
        amgt.set_level_policy([])
    return log, out


@pytest.mark.parametrize("what", ["header", "columns", "values", "multi"])
def test_no_memory_for_a_copy_keeps_the_blocks(amgt, orc, what):
    """The copies are optional: when the allocator has no memory for a part
    of A_0's (its slice headers, columns or values), the setup goes on
    and the products run on the blocks; when it has none for the vectors of
    a multi-right-hand-side solve while copies are held, they are given back
    and the solve goes on.  Same iterations and solutions to 1e-9."""
    dims = (60, 58, 56)
    A, Ps = orc.laplacian(*dims), orc.geometric_hierarchy(*dims)
    b = torch.from_numpy(A.to_scipy() @ orc.rand_uniform(6, A.n)).cuda()
    # A_0's copy: slices of 32 rows, 16-bit offsets, 8-byte values; its headers
    # are the first ones made
    hdr, columns, values = 16 * -(-A.m // 32), 2 * 32 * sliced_steps(A), 8 * 32 * sliced_steps(A)
    log, ref = _solve_all(amgt, A, Ps, b, multi=what == "multi")
    assert log.sizes.count(columns) == log.sizes.count(values) == 1
    fail = {"header": lambda s: s[-1] == hdr and s.count(hdr) == 1, "columns": lambda s: s[-1] == columns,
            "values": lambda s: s[-1] == values,
            "multi": lambda s: s[-1] == 8 * 2 * A.n and s.count(8 * 2 * A.n) == 1}[what]  # the first multivector
    log, out = _solve_all(amgt, A, Ps, b, fail, what == "multi")
    assert log.failed == 1
    for (x, it, rel), (x0, it0, _) in zip(out, ref):
        assert it == it0 and rel <= 1e-8
        assert torch.linalg.norm(x - x0) <= 1e-9 * torch.linalg.norm(x0)
