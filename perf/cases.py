"""Timed cases of the mBSR framework: the calls a multigrid user makes.

One case is one pass through a public entry point (or the few calls that
make one step of a user's program) on a problem that the configurations, the
tests and the benchmark of this repository use: structured 5-, 7- and
27-point operators in 2D and 3D, linear and BoomerAMG interpolation.  Small
grids are where launches and latency count, the 128^3 ones where bytes do;
odd extents give ragged 4x4 blocks.  Inputs are made on the GPU from the
seed (right-hand sides, vectors, the coefficients of the variable-coefficient
operators).

Fields of a case: op, the grid (nx, ny, nz), the operator (pts: 5, 7, 27;
27 with coef = "var" has log-normal coefficients), prec (0 fp64, 1 fp32,
2 fp16, 3 bf16), nvec, beta, interp ("linear", "boomer").
"""
import functools
import math
import random

import numpy as np
import torch

import amgt_b200 as amgt
from amgt_b200 import boomer, problems
from amgt_b200.amg import AmgSolver, BatchSolver, default_params

MIXED = [0, 1, 1, 2]  # level 0 fp64, levels 1-2 fp32, deeper levels fp16
FGMRES = dict(flexible=1, smooth_prec0=1, galerkin_by_level=1, solver=1, restart=30, inner_prec0=1, inner_tol=1e-4)


def listed():
    return [
        # the smallest call: HYPRE's matvec hook on the 2D 128x128 operator (config 1), launch latency
        {"name": "matvec_hook_2d128", "op": "hook", "nx": 128, "ny": 128, "nz": 1, "pts": 5, "coef": "one",
         "prec": 0, "beta": 0.0},
        # the benchmark's headline: fp64 SpMV of the 7-point 128^3 operator (smoothing and residuals of a solve)
        {"name": "spmv_7pt128", "op": "spmv", "nx": 128, "ny": 128, "nz": 128, "pts": 7, "coef": "one", "prec": 0,
         "beta": 0.0},
        # a middle level's fp32 product on a dense stencil with odd extents (ragged last blocks)
        {"name": "spmv_27pt_odd_fp32", "op": "spmv", "nx": 95, "ny": 97, "nz": 93, "pts": 27, "coef": "var", "prec": 1,
         "beta": 0.0},
        # many right-hand sides: 32 vectors times the 7-point 64^3 operator (the batching configuration's hot op)
        {"name": "spmm_7pt64_32", "op": "spmm", "nx": 64, "ny": 64, "nz": 64, "pts": 7, "coef": "one", "prec": 1,
         "nvec": 32},
        # entry of every matrix: CSR -> mBSR of the 27-point variable-coefficient 96^3 operator
        {"name": "csr2bsr_27pt96", "op": "convert", "nx": 96, "ny": 96, "nz": 96, "pts": 27, "coef": "var"},
        # one level of a setup: transpose and Galerkin product at 128^3 (the benchmark's level 0)
        {"name": "galerkin_7pt128", "op": "galerkin", "nx": 128, "ny": 128, "nz": 128, "pts": 7, "coef": "one",
         "prec": 0},
        # HYPRE's SpGEMM benchmark product A*A through its hook, 27-point
        {"name": "square_27pt", "op": "square", "nx": 72, "ny": 64, "nz": 80, "pts": 27, "coef": "one"},
        # whole solves: setup + solve to 1e-8 with BoomerAMG's interpolation, 2D (latency) and 3D (bytes)
        {"name": "amg_2d128", "op": "amg", "nx": 128, "ny": 128, "nz": 1, "pts": 5, "coef": "one",
         "interp": "boomer", "mixed": False},
        {"name": "amg_7pt128", "op": "amg", "nx": 128, "ny": 128, "nz": 128, "pts": 7, "coef": "one",
         "interp": "boomer", "mixed": False},
        # the mixed-precision configuration: FGMRES(30) with refinement on the 27-point 96^3 operator
        {"name": "amg_27pt96_mixed", "op": "amg", "nx": 96, "ny": 96, "nz": 96, "pts": 27, "coef": "var",
         "interp": "linear", "mixed": True},
        # 32 right-hand sides on one hierarchy (the handle is kept), mixed precision
        {"name": "multirhs_7pt64_32", "op": "multi", "nx": 64, "ny": 64, "nz": 64, "pts": 7, "coef": "one",
         "nvec": 32},
        # 64 uneven 2D systems at once: setup + solve
        {"name": "batch_2d_64", "op": "batch", "systems": 64, "side_min": 32, "side_max": 512, "sides_seed": 0},
    ]


def _grid(rng, lo, hi, pts):
    """Extents with lo..hi unknowns (log-uniform), odd ones as likely as even ones."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    d = 2 if pts == 5 else 3
    side = n ** (1.0 / d)
    a, b = side * rng.uniform(0.8, 1.25), side * rng.uniform(0.8, 1.25)
    dims = [a, b] if d == 2 else [a, b, n / (a * b)]
    if d == 2:
        dims[1] = n / a
    dims = [max(4, int(x)) for x in dims]
    while math.prod(dims) > hi:
        dims[dims.index(max(dims))] -= 1
    return {"nx": dims[0], "ny": dims[1], "nz": dims[2] if d == 3 else 1}


def draw(rng):
    op = rng.choice(["hook", "spmv", "spmv", "spmm", "convert", "galerkin", "square", "amg", "amg", "amg", "multi",
                     "batch"])
    if op == "batch":
        lo = rng.randint(16, 128)
        return {"op": op, "systems": rng.randint(3, 64), "side_min": lo, "side_max": rng.randint(lo, 512),
                "sides_seed": rng.randint(0, 1 << 30)}
    pts = rng.choice([5, 7, 27])
    c = {"op": op, "pts": pts, "coef": rng.choice(["one", "var"]) if pts == 27 else "one"}
    if op in ("hook", "spmv"):
        c.update(_grid(rng, 1000, 800_000 if pts == 27 else 2_000_000, pts))
        c["prec"] = 0 if op == "hook" else rng.choice([0, 0, 1, 2, 3])
        c["beta"] = rng.choice([0.0, 0.0, 1.0])
    elif op == "spmm":
        c.update(_grid(rng, 1000, 80_000 if pts == 27 else 260_000, pts))
        c["prec"], c["nvec"] = rng.choice([0, 1, 1, 2, 3]), rng.choice([1, 4, 8, 13, 16, 27, 32])
    elif op == "convert":
        c.update(_grid(rng, 1000, 800_000 if pts == 27 else 2_000_000, pts))
    elif op == "galerkin":
        c.update(_grid(rng, 1000, 400_000 if pts == 27 else 2_000_000, pts))
        c["prec"] = rng.choice([0, 0, 1, 2])
    elif op == "square":
        c.update(_grid(rng, 1000, 300_000 if pts == 27 else 1_000_000, pts))
    elif op == "amg":
        c["mixed"] = rng.random() < 0.4
        c["interp"] = "linear" if c["mixed"] or c["coef"] == "var" else rng.choice(["linear", "boomer"])
        top = 200_000 if c["interp"] == "boomer" else (700_000 if pts == 27 else 1_500_000)
        c.update(_grid(rng, 2000, top, pts))
    else:
        c.update(_grid(rng, 2000, 60_000 if pts == 27 else 250_000, pts))
        c["nvec"] = rng.choice([2, 8, 16, 21, 32])
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(seed, *shape):
    """Uniform in [-1, 1)."""
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=_gen(seed)) * 2.0 - 1.0


def _csr(cols, vals, valid):
    """Candidate entries (n, k) in storage order -> device CSR arrays."""
    ia = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(valid.sum(dim=1), 0, out=ia[1:])
    return ia.int(), cols[valid].int().contiguous(), vals[valid].contiguous()


def _coords(nx, ny, nz):
    r = torch.arange(nx * ny * nz, dtype=torch.int64, device="cuda")
    return r, r % nx, (r // nx) % ny, r // (nx * ny)


def _offsets(pts):
    if pts == 27:
        box = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        return [o for o in box if o != (0, 0, 0)]
    line = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    return [o for o in line if pts == 7 or o[2] == 0]


def _operator(case, seed):
    """The operator as a device CSR tuple (diagonal first, the rest ascending, as HYPRE's generators store it) and
    its candidate arrays (cols, vals with 0 outside the domain).  coef "var": node coefficients exp(2 N(0, 1)) with
    a ratio of 1e3, couplings their harmonic means (as problems.varcoef27)."""
    nx, ny, nz, pts = case["nx"], case["ny"], case["nz"], case["pts"]
    n = nx * ny * nz
    r, x, y, z = _coords(nx, ny, nz)
    var = case["coef"] == "var"
    offs = _offsets(pts)
    if var:
        clip = 0.5 * math.log(1e3)
        g = torch.randn(n, dtype=torch.float64, device="cuda", generator=_gen(seed + 7919))
        kap = torch.exp(torch.clamp(2.0 * g, -clip, clip))
    cols, vals, valid = [r], [None], [torch.ones(n, dtype=torch.bool, device="cuda")]
    diag = torch.zeros(n, dtype=torch.float64, device="cuda")
    for dx, dy, dz in offs:
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
        c = torch.where(ok, r + dx + nx * (dy + ny * dz), r)
        h = torch.ones(n, dtype=torch.float64, device="cuda")
        if var:
            w = 2.0 ** (1 - abs(dx) - abs(dy) - abs(dz))
            h = w * 2.0 * kap * kap[c] / (kap + kap[c])
        diag += h
        cols.append(c)
        vals.append(torch.where(ok, -h, torch.zeros_like(h)))
        valid.append(ok)
    vals[0] = diag
    cols, vals, valid = torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(valid, 1)
    return (n, n) + _csr(cols, vals, valid), (cols, vals)


def _times(cand, x):
    """A x from the candidate arrays, in a fixed order; x: (n,) or (n, nvec)."""
    cols, vals = cand
    out = torch.zeros_like(x)
    for k in range(cols.shape[1]):
        v = vals[:, k] if x.dim() == 1 else vals[:, k, None]
        out += v * x[cols[:, k]]
    return out


def _interp_1d(i, fine):
    """Two (coarse index, weight, valid) candidates per fine index of a vertex-centred axis."""
    if fine == 1:
        o = torch.ones(i.shape, dtype=torch.float64, device="cuda")
        t = torch.ones(i.shape, dtype=torch.bool, device="cuda")
        return [(i * 0, o, t), (i * 0, 0 * o, ~t)]
    nc = (fine + 1) // 2
    odd = (i & 1) == 1
    second = odd & ((i + 1) // 2 < nc)
    return [(i // 2, torch.where(odd, 0.5, 1.0).double(), torch.ones_like(odd)),
            (torch.where(second, (i + 1) // 2, 0), torch.where(second, 0.5, 0.0).double(), second)]


def _interp(nx, ny, nz):
    """Linear interpolation to every second grid point (device CSR) and the coarse extents (as problems.interp)."""
    cd = tuple((d + 1) // 2 if d > 1 else 1 for d in (nx, ny, nz))
    _, x, y, z = _coords(nx, ny, nz)
    px, py, pz = _interp_1d(x, nx), _interp_1d(y, ny), _interp_1d(z, nz)
    cols, vals, valid = [], [], []
    for cz in pz:
        for cy in py:
            for cx in px:
                cols.append(cx[0] + cd[0] * (cy[0] + cd[1] * cz[0]))
                vals.append(cx[1] * cy[1] * cz[1])
                valid.append(cx[2] & cy[2] & cz[2])
    return (nx * ny * nz, math.prod(cd)) + _csr(torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(valid, 1)), cd


def _linear_hierarchy(dims, coarse_rows=64):
    Ps = []
    while math.prod(dims) > coarse_rows:
        P, cd = _interp(*dims)
        if cd == dims:
            break
        Ps.append(P)
        dims = cd
    return Ps


@functools.lru_cache(maxsize=3)
def _boomer_host(nx, ny, nz, pts):
    """Interpolation operators of HYPRE's host BoomerAMG setup for the constant-coefficient operator (host arrays)."""
    n, _, ia, ja, a = problems.box(nx, ny, nz) if pts == 27 else problems.laplacian(nx, ny, nz)
    Ps, _ = boomer.hypre_hierarchy((a, ja, ia))
    out = []
    for P in Ps:
        P.sort_indices()
        out.append((P.shape[0], P.shape[1], P.indptr.astype(np.int32), P.indices.astype(np.int32), P.data))
    return out


def _boomer_hierarchy(case):
    return [P[:2] + tuple(torch.from_numpy(v).cuda() for v in P[2:])
            for P in _boomer_host(case["nx"], case["ny"], case["nz"], case["pts"])]


def _sides(case):
    r = random.Random(case["sides_seed"])
    return [r.randint(case["side_min"], case["side_max"]) for _ in range(case["systems"])]


def _interps(case):
    if case.get("interp") == "boomer":
        return _boomer_hierarchy(case)
    return _linear_hierarchy((case["nx"], case["ny"], case["nz"]))


def prepare(case, seed):
    op = case["op"]
    amgt.set_level_policy([0])
    if op == "batch":
        systems, b = [], []
        for k, side in enumerate(_sides(case)):
            A, cand = _operator({"nx": side, "ny": side, "nz": 1, "pts": 5, "coef": "one"}, 0)
            systems.append((A, _linear_hierarchy((side, side, 1))))
            b.append(_times(cand, _uniform(1000 * seed + k, side * side)))
        return {"op": op, "systems": systems, "b": torch.cat(b)}
    A, cand = _operator(case, seed)
    n = A[0]
    st = {"op": op, "case": case, "A": A}
    if op == "hook":
        st["M"] = amgt.CSRMatrix.create(*A)
        st["x"], st["y0"] = _uniform(seed, n), _uniform(seed + 1, n)
        st["y"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    elif op == "spmv":
        st["M"] = amgt.Bsr.from_csr(*A)
        if case["prec"]:
            st["M"].make_shadow(case["prec"])
        st["x"], st["y0"] = _uniform(seed, n), _uniform(seed + 1, n)
        st["y"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    elif op == "spmm":
        st["M"] = amgt.Bsr.from_csr(*A)
        st["M"].make_exact()
        if case["prec"]:
            st["M"].make_shadow(case["prec"])
        st["x"] = _uniform(seed, n, case["nvec"])
        st["y"] = torch.zeros(n, case["nvec"], dtype=torch.float64, device="cuda")
    elif op == "galerkin":
        st["M"] = amgt.Bsr.from_csr(*A)
        P, _ = _interp(case["nx"], case["ny"], case["nz"])
        # smooth positive weights instead of the constant ones: other values for another seed
        st["Pcsr"] = P[:4] + (P[4] * (1.0 + 0.25 * _uniform(seed + 2, P[4].numel())),)
        st["P"] = amgt.Bsr.from_csr(*st["Pcsr"])
    elif op == "square":
        st["A"] = A[:4] + (A[4] * (1.0 + 0.25 * _uniform(seed + 2, A[4].numel())),)
        st["M"] = amgt.CSRMatrix.create(*st["A"])
    elif op == "amg":
        st["Ps"] = _interps(case)
        st["b"] = _times(cand, _uniform(seed, n))
    elif op == "multi":
        Ps = _interps(case)
        amgt.set_level_policy(MIXED)
        st["S"] = AmgSolver(A, Ps, default_params(inner_prec0=1, galerkin_by_level=1))
        st["b"] = _times(cand, _uniform(seed, n, case["nvec"]))
    return st


# --------------------------------------------------------------------- pass
def run(state):
    op, case = state["op"], state.get("case")
    if op == "hook":
        y = state["y"]
        if case["beta"]:
            y.copy_(state["y0"])
        amgt.hypre_CSRMatrixMatvecCusparseNewAPI(0, 1.0, state["M"], state["x"], case["beta"], y)
        return y
    if op == "spmv":
        y = state["y"]
        if case["beta"]:
            y.copy_(state["y0"])
        return state["M"].spmv(state["x"], y, alpha=1.0, beta=case["beta"], prec=case["prec"])
    if op == "spmm":
        return state["M"].spmm_rm(state["x"], state["y"], prec=case["prec"])
    if op == "convert":
        state["out"] = B = amgt.Bsr.from_csr(*state["A"])  # kept: the arrays belong to it
        return {"ptr": B.ptr(), "idx": B.idx(), "map": B.map(), "val": B.val()}
    if op == "galerkin":
        R = state["P"].transpose()
        AP, _ = amgt.spgemm(state["M"], state["P"], prec=case["prec"], want_csr=False)
        C, csr = amgt.spgemm(R, AP, prec=case["prec"], want_csr=True)
        state["out"] = (C, csr)
        return {"ptr": C.ptr(), "idx": C.idx(), "map": C.map(), "val": C.val(), "ia": csr.ia, "ja": csr.ja,
                "a": csr.a}
    if op == "square":
        state["out"] = C = amgt.hypreDevice_CSRSpGemm(state["M"], state["M"])
        return {"ia": C.i, "ja": C.j, "a": C.data}
    if op == "amg":
        amgt.set_level_policy(MIXED if case["mixed"] else [0])
        S = AmgSolver(state["A"], state["Ps"], default_params(**FGMRES) if case["mixed"] else default_params())
        x, _, _ = S.solve(state["b"])
        S.free()
        return x
    if op == "multi":
        amgt.set_level_policy(MIXED)
        X, _, _ = state["S"].solve_multi(state["b"])
        return X
    amgt.set_level_policy([0])
    S = BatchSolver(state["systems"], default_params())
    x, _, _, _ = S.solve_batch(state["b"])
    S.free()
    return x


# --------------------------------------------------------------------- work
def _nnz(nx, ny, nz, pts):
    return nx * ny * nz + sum((nx - abs(a)) * (ny - abs(b)) * (nz - abs(c)) for a, b, c in _offsets(pts))


def _blocks(nx, ny, nz, pts):
    """4x4 blocks of a stencil operator: a stencil line with x neighbours touches three block columns, one without
    them one (two when the line's offset is not a multiple of 4)."""
    lines = {}
    for a, b, c in _offsets(pts) + [(0, 0, 0)]:
        lines.setdefault((b, c), set()).add(a)
    total = 0.0
    for (b, c), xs in lines.items():
        per = 3.0 if len(xs) > 1 else (1.0 if (nx * (b + ny * c)) % 4 == 0 else 2.0)
        total += per * nx * (ny - abs(b)) * (nz - abs(c)) / 4.0
    return total


def _cycle_work(nnz, complexity, n, rows, iters):
    """One solve: per iteration two operator passes per level and one more on the finest, one pass over each
    transfer both ways (about four entries a row), 12 bytes an entry, and six vectors per row and level; once the
    CSR inputs and the hierarchy."""
    entries = iters * (nnz * (2.0 * complexity + 1.0) + 8.0 * rows * n)
    vec = 8.0 * 6.0 * iters * rows * n
    setup = 12.0 * nnz * complexity + 12.0 * 4.0 * rows * n
    return {"bytes": 12.0 * entries + vec + setup, "flops": 2.0 * entries}


def work(case):
    op = case["op"]
    if op == "batch":
        n = sum(s * s for s in _sides(case))
        return _cycle_work(5.0 * n, 1.8, n, 1.34, 13)
    dims = (case["nx"], case["ny"], case["nz"])
    pts, n = case["pts"], math.prod(dims)
    nnz, nb = _nnz(*dims, pts), _blocks(*dims, pts)
    vb = {0: 8, 1: 4, 2: 2, 3: 2}[case.get("prec", 0)]
    if op in ("hook", "spmv"):
        return {"bytes": nb * (16 * vb + 4) + n + 16 * n + (8 * n if case["beta"] else 0), "flops": 2 * nnz}
    if op == "spmm":
        if case["coef"] == "one":
            vb = min(vb, 2)  # the values are whole numbers: exact in fp16
        return {"bytes": nb * (16 * vb + 4) + n + 16 * n * case["nvec"], "flops": 2 * nnz * case["nvec"]}
    if op == "convert":
        return {"bytes": 12 * nnz + 4 * n + nb * (128 + 6) + n, "flops": 0}
    three = dims[2] > 1
    if op == "galerkin":
        cd = tuple((d + 1) // 2 if d > 1 else 1 for d in dims)
        pnnz = n * (27 / 8 if three else 9 / 4)
        cn, cp = math.prod(cd), 27 if three else 9
        cnb = _blocks(*cd, 27) if three else 9 / 4 * cn
        pb = pnnz / 4.1
        return {"bytes": nb * (16 * vb + 6) + 2 * pb * (16 * vb + 6) + cnb * 134 + cn * cp * 12,
                "flops": 2 * (nnz * pnnz / n + pnnz * cp / 4)}
    if op == "square":
        per = {5: 13, 7: 25, 27: 125}[pts]
        return {"bytes": nb * 134 + per * n * 12 + per * n / 16 / 0.4 * 134, "flops": 2 * nnz * nnz / n}
    if op == "amg":
        oc = 1.3 if case["interp"] == "linear" else (3.3 if three else 2.3)
        rows = 1.15 if case["interp"] == "linear" and three else 1.6
        return _cycle_work(nnz, oc, n, rows, 13)
    w = _cycle_work(nnz, 1.5, n, 1.15, 1)
    return {"bytes": 16 * (w["bytes"] + 8 * 1.15 * n * 12 * case["nvec"]), "flops": 16 * w["flops"] * case["nvec"]}


def tolerance(case):
    """About four times what the same sums in another order (other lanes per row) give."""
    op, prec = case["op"], case.get("prec", 0)
    if op == "convert":
        return "exact"  # values are moved, not computed
    if op in ("amg", "batch", "multi"):
        # x at a relative residual of 1e-8, itself about 1e-8 from the exact solution: fp64 iterates agree to 5e-14
        # (2D, 1.1M rows); with reduced levels two roundings differ by up to 7e-10, and a correction that stops one
        # inner step apart by the error that is left
        if op == "multi" or case.get("mixed", False):
            return {"rel": 1e-8, "max": 4e-8}
        return {"rel": 4e-13, "max": 2e-12}
    if op == "galerkin" and prec == 2:
        return {"rel": 2e-5, "max": 2e-3}  # A P is rounded to fp16 between the two products: a last bit may flip
    if op == "spmm" and prec:
        return {"rel": 6e-7, "max": 6e-6}  # fp32 sums, or tf32 with a high / low split
    if prec:
        return {"rel": 4e-7, "max": 3e-6}  # fp32 sums
    return {"rel": 1e-15, "max": 2e-14}


# -------------------------------------------------------------------- exact
def _sparse(M):
    return torch.sparse_csr_tensor(M[2].long(), M[3].long(), M[4], size=(M[0], M[1]))


def _sorted_csr(C):
    ia, ja, a = C.crow_indices(), C.col_indices(), C.values()
    rows = torch.repeat_interleave(torch.arange(C.shape[0], device="cuda"), ia[1:] - ia[:-1])
    key, order = torch.sort(rows * C.shape[1] + ja)
    return key // C.shape[1], key % C.shape[1], a[order]


def _block_values(rows, cols, a, ncols):
    nbc = (ncols + 3) // 4
    _, blk = torch.unique((rows // 4) * nbc + cols // 4, return_inverse=True)
    val = torch.zeros(16 * (int(blk.max()) + 1), dtype=torch.float64, device="cuda")
    val[16 * blk + 4 * (rows % 4) + cols % 4] = a
    return val


def exact(case, seed):
    op = case["op"]
    if op == "convert":
        return None
    if op == "batch":
        return torch.cat([_uniform(1000 * seed + k, s * s) for k, s in enumerate(_sides(case))])
    n = case["nx"] * case["ny"] * case["nz"]
    if op == "amg":
        return _uniform(seed, n)
    if op == "multi":
        return _uniform(seed, n, case["nvec"])
    A, cand = _operator(case, seed)
    if op in ("hook", "spmv"):
        y = _times(cand, _uniform(seed, n))
        return y + _uniform(seed + 1, n) if case["beta"] else y
    if op == "spmm":
        return _times(cand, _uniform(seed, n, case["nvec"]))
    if op == "square":
        S = _sparse(A[:4] + (A[4] * (1.0 + 0.25 * _uniform(seed + 2, A[4].numel())),))
        _, _, a = _sorted_csr(S @ S)
        return {"ia": None, "ja": None, "a": a}
    P, _ = _interp(case["nx"], case["ny"], case["nz"])
    P = _sparse(P[:4] + (P[4] * (1.0 + 0.25 * _uniform(seed + 2, P[4].numel())),))
    AP = _sparse(A) @ P
    pr = torch.repeat_interleave(torch.arange(n, device="cuda"), P.crow_indices()[1:] - P.crow_indices()[:-1])
    pc, order = torch.sort(P.col_indices(), stable=True)
    ra = torch.zeros(P.shape[1] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(pc, minlength=P.shape[1]), 0, out=ra[1:])
    R = torch.sparse_csr_tensor(ra, pr[order], P.values()[order], size=(P.shape[1], n))
    rows, cols, a = _sorted_csr(R @ AP)
    return {"ptr": None, "idx": None, "map": None, "val": _block_values(rows, cols, a, P.shape[1]), "ia": None,
            "ja": None, "a": a}
