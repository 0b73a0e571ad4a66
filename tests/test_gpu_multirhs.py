"""GPU tests of the fused multi-right-hand-side products (spmm_tc.cu's
CUDA-core form and its epilogues), at the column counts where its lanes and
access widths change: 1 and 7 (scalar accesses), 12 (8 lanes a block row), 24
(16 lanes, strides known at run time), 32 (constant strides)."""
import numpy as np
import pytest
import torch

from gpu_util import random_csr, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 7, 12, 24])
@pytest.mark.parametrize("policy,inner", [([0], 0), ([0, 1, 2], 1)])
def test_solve_multi_column_counts(amgt, orc, nv, policy, inner):
    """Each column reaches 1e-8, checked in fp64, with x within 1e-6 of the
    oracle's fp64 solve (both stop at a relative residual of 1e-8)."""
    from amgt_b200.amg import AmgSolver, default_params

    dims = (23, 19, 14)
    A, Ps = orc.varcoef27(*dims, seed=2), orc.geometric_hierarchy(*dims)
    B = np.ascontiguousarray(np.stack([orc.rand_uniform(v, A.n) for v in range(nv)], axis=1))
    amgt.set_level_policy(policy)
    try:
        S = AmgSolver(to_dev(A), [to_dev(P) for P in Ps], default_params(inner_prec0=inner))
        X, its, rel = S.solve_multi(torch.from_numpy(B).cuda())
        S.free()
    finally:
        amgt.set_level_policy([])
    X, Sa, H = X.cpu().numpy(), A.to_scipy(), orc.Amg(A, Ps)
    for v in range(nv):
        assert np.linalg.norm(B[:, v] - Sa @ X[:, v]) <= 1.0000001e-8 * np.linalg.norm(B[:, v])
        xo = H.solve(B[:, v])[0]
        assert np.linalg.norm(X[:, v] - xo) <= 1e-6 * np.linalg.norm(xo)


@pytest.mark.parametrize("nvec", [2, 8, 24, 31])
@pytest.mark.parametrize("prec", [0, 1])
def test_spmm_without_bitmaps_and_misaligned(amgt, orc, nvec, prec):
    """A caller's amgt_bsr without bitmaps takes full blocks (bounded by the
    column count), and X / Y off 16-byte alignment take scalar accesses; per
    row 1e-12 (fp64) or 1e-5 (fp32 sums) of |A||x|."""
    import ctypes

    A = random_csr(orc, 211, 173, 9, seed=8)
    R = orc.csr2bsr(A)
    G = amgt.Bsr.from_csr(*to_dev(A))
    if prec:
        G.make_shadow(prec)
    keep = G.s.blcMap
    X = np.ascontiguousarray(np.stack([orc.rand_uniform(10 + v, A.n) for v in range(nvec)], axis=1))
    xb = torch.zeros(A.n * nvec + 1, dtype=torch.float64, device="cuda")
    yb = torch.zeros(A.m * nvec + 1, dtype=torch.float64, device="cuda")
    xb[1:] = torch.from_numpy(X.ravel()).cuda()
    G.s.blcMap = None
    try:
        rc = amgt.lib().amgt_spmm_rm(prec, 1, 1.0, ctypes.byref(G.s), nvec, xb[1:].data_ptr(), 0.0,
                                     yb[1:].data_ptr(), None)
        torch.cuda.synchronize()
    finally:
        G.s.blcMap = keep
    assert rc == 0
    got = yb[1:].cpu().numpy().reshape(A.m, nvec)
    for v in range(nvec):
        want = orc.spmv(R, X[:, v], prec=prec)
        assert np.all(np.abs(got[:, v] - want) <= (1e-12 if prec == 0 else 1e-5) * orc.spmv_bound(R, X[:, v], None) + 1e-300)


@pytest.mark.parametrize("nvec", [1, 2, 5, 8, 13, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("dims,pts", [((5, 3, 1), 7), ((19, 11, 9), 27), ((47, 31, 29), 7), ((55, 53, 54), 7)])
def test_spmm_cuda_core_forms(amgt, orc, dims, pts, nvec):
    """The CUDA-core form where its lanes per block row, its parts of a block
    row (8, 4, 2, 1 from 4 to 40,000 block rows) and its access widths change,
    at fp64, fp32 and fp16 values, beta 0 and not: per row 1e-12 (fp64) or
    1e-5 (fp32 sums of about 27 terms) of |A||x| + |y|."""
    T = orc.laplacian(*dims) if pts == 7 else orc.box(*dims)
    A = orc.CSR(T.m, T.n, T.ia, T.ja, np.random.default_rng(2).uniform(-1, 1, T.ja.size))
    G = amgt.Bsr.from_csr(*to_dev(A))
    X = np.ascontiguousarray(np.stack([orc.rand_uniform(v, A.n) for v in range(nvec)], axis=1))
    Y0 = np.ascontiguousarray(np.stack([orc.rand_uniform(50 + v, A.m) for v in range(nvec)], axis=1))
    x = torch.from_numpy(X).cuda()
    S = A.to_scipy()
    for prec, beta in ((0, 0.0), (0, -0.5), (1, 0.0), (2, -0.5)):
        if prec:
            G.make_shadow(prec)
        M = S.copy()
        if prec:
            M.data = M.data.astype(np.float32 if prec == 1 else np.float16).astype(np.float64)
        y = torch.from_numpy(Y0).cuda()
        G.spmm_rm(x, y, alpha=1.5, beta=beta, prec=prec, engine=1)
        want = 1.5 * (M @ X) + beta * Y0
        bound = 1.5 * (abs(M) @ np.abs(X)) + np.abs(beta * Y0)
        err = np.abs(y.cpu().numpy() - want)
        assert np.all(err <= (1e-12 if prec == 0 else 1e-5) * bound + 1e-300)
