"""GPU tests with infinities and NaN."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("holes", [False, True])
def test_nan_right_hand_side_stays_in_its_system(amgt, orc, holes):
    """62 systems of 56 x 37 unknowns and two coarse levels: all sizes (2,072,
    532, 140) are multiples of 4, so no block holds two systems, but not of
    32, so slices of the sliced copies do.  A NaN in one system's right-hand
    side (whose last slice holds rows of the next one) changes no bit of the
    others' solutions; also with empty rows in the interpolation."""
    from amgt_b200.amg import BatchSolver, default_params

    ns, bad = 62, 40
    A, Ps = orc.laplacian(56, 37, 1), orc.geometric_hierarchy(56, 37, 1)[:2]
    n, P = A.n, Ps[0]
    if holes:  # unknowns 0 .. 7 and 9 are not interpolated
        keep = np.ones(n, bool)
        keep[[0, 1, 2, 3, 4, 5, 6, 7, 9]] = False
        lens = np.where(keep, np.diff(P.ia), 0)
        sel = np.repeat(keep, np.diff(P.ia))
        Ps[0] = orc.CSR(P.m, P.n, np.concatenate([[0], np.cumsum(lens)]).astype(np.int32), P.ja[sel], P.a[sel])
    amgt.set_level_policy([0])
    try:
        S = BatchSolver([(to_dev(A), [to_dev(P) for P in Ps])] * ns, default_params(max_coarse_rows=16384))
        assert ns * orc.csr2bsr(Ps[0]).nblk >= 65536  # A_0 and P_0 are copied
        assert n % 32 != 0 and all(k % 4 == 0 for k in (n, Ps[0].n, Ps[1].n))
        b = torch.from_numpy(orc.rand_uniform(5, ns * n)).cuda()
        x0, it0, rel0, _ = S.solve_batch(b)
        b[bad * n + 7] = float("nan")
        x1, it1, rel1, _ = S.solve_batch(b)
        S.free()
    finally:
        amgt.set_level_policy([])
    assert max(rel0) <= 1e-8
    for s in range(ns):
        if s == bad:
            continue
        sl = slice(s * n, (s + 1) * n)
        assert torch.equal(x0[sl], x1[sl]) and it0[s] == it1[s] and rel0[s] == rel1[s], s


@pytest.mark.parametrize("nvec", [1, 7, 8, 16, 24, 32])
@pytest.mark.parametrize("prec", [0, 1])
def test_spmm_keeps_a_stored_infinity(amgt, orc, nvec, prec):
    """Block rows of 1 to 8 blocks whose last block holds an infinity: its
    row's result is that infinity (x > 0), every other row's is as without
    it."""
    import scipy.sparse as sp

    nb = 48
    rows, cols, vals = [], [], []
    rng = np.random.default_rng(3)
    for b in range(nb):
        k = 1 + b % 8
        for j in range(k):
            for r in range(4):
                rows.append(4 * b + r), cols.append(4 * ((b + 5 * j) % nb) + (r + j) % 4), vals.append(rng.uniform(0.5, 1))
    S = sp.csr_matrix((vals, (rows, cols)), shape=(4 * nb, 4 * nb))
    S.sort_indices()
    A = orc.CSR(4 * nb, 4 * nb, S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data.copy())
    last = A.ia[1:] - 1  # row r's last entry lies in its block row's last block
    X = 0.5 + np.ascontiguousarray(np.stack([np.abs(orc.rand_uniform(v, A.n)) for v in range(nvec)], axis=1))
    hit = np.arange(0, A.m, 4) + np.arange(nb) % 4  # one row per block row
    a = A.a.copy()
    a[last[hit]] = np.inf
    out = []
    for v in (A.a, a):
        G = amgt.Bsr.from_csr(*to_dev(orc.CSR(A.m, A.n, A.ia, A.ja, v)))
        if prec:
            G.make_shadow(prec)
        out.append(G.spmm_rm(torch.from_numpy(X).cuda(), prec=prec, engine=1).cpu().numpy())
    other = np.setdiff1d(np.arange(A.m), hit)
    assert np.all(out[1][hit] == np.inf)
    np.testing.assert_array_equal(out[1][other], out[0][other])


@pytest.mark.parametrize("prec", [0, 1, 2, 3])
@pytest.mark.parametrize("kernel", ["staged", "wide"])
def test_spgemm_nonfinite_entries_meet_unstored_ones(amgt, orc, kernel, prec):
    """A block product multiplies unstored entries as zeros, so an infinity
    of B against an unstored entry of A gives NaN, and one of A against an
    unstored entry of B too, whichever of the staged and the wide-row kernel
    the sizes pick: the kinds of all C values equal those of dense 4x4 block
    products (which of them are infinite or NaN does not depend on the order
    of sums of one sign)."""
    T = orc.laplacian(64, 32, 20) if kernel == "staged" else orc.box(40, 40, 24)
    rng = np.random.default_rng(21)
    a, b = (np.abs(rng.uniform(0.5, 1, T.ja.size)) for _ in range(2))
    a[rng.integers(0, a.size, 3)] = np.inf
    b[rng.integers(0, b.size, 5)] = np.inf
    b[rng.integers(0, b.size, 2)] = np.nan
    A, B = orc.CSR(T.m, T.n, T.ia, T.ja, a), orc.CSR(T.m, T.n, T.ia, T.ja, b)
    GA, GB = amgt.Bsr.from_csr(*to_dev(A)), amgt.Bsr.from_csr(*to_dev(B))
    if prec:
        GA.make_shadow(prec), GB.make_shadow(prec)
    GC, csr = amgt.spgemm(GA, GB, prec=prec)
    c = GC.host()
    lens = np.diff(c["bptr"])  # enough block rows for these two kernels, and the rule between them
    assert lens.size >= 64 * torch.cuda.get_device_properties(0).multi_processor_count
    assert (lens.mean() > 48 and lens.max() > 64) == (kernel == "wide")
    RA, RB = orc.csr2bsr(A), orc.csr2bsr(B)
    # only block rows that a non-finite block reaches can hold a non-finite value
    va, vb = RA.bval.reshape(-1, 4, 4), RB.bval.reshape(-1, 4, 4)
    brow = np.repeat(np.arange(RA.bptr.size - 1), np.diff(RA.bptr))
    badb = np.unique(np.repeat(np.arange(RB.bptr.size - 1), np.diff(RB.bptr))[~np.isfinite(vb).all((1, 2))])
    hit = np.unique(brow[~np.isfinite(va).all((1, 2)) | np.isin(RA.bidx, badb)])
    got = c["bval"].reshape(-1, 4, 4)
    finite = np.ones(got.shape[0], bool)
    for i in hit:
        C = {}
        with np.errstate(invalid="ignore"):
            for p in range(RA.bptr[i], RA.bptr[i + 1]):
                k = RA.bidx[p]
                for q in range(RB.bptr[k], RB.bptr[k + 1]):
                    j = RB.bidx[q]
                    C[j] = C.get(j, 0.0) + (va[p][:, :, None] * vb[q][None, :, :]).sum(1)
        for t in range(c["bptr"][i], c["bptr"][i + 1]):
            finite[t] = False
            want = C[c["bidx"][t]]
            np.testing.assert_array_equal(np.isnan(got[t]), np.isnan(want), err_msg=f"block row {i}")
            np.testing.assert_array_equal(np.isinf(got[t]), np.isinf(want), err_msg=f"block row {i}")
    assert hit.size > 0 and np.isfinite(got[finite]).all()
