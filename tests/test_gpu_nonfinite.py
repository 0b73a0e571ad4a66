"""GPU tests with infinities and NaN."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


def test_nan_right_hand_side_stays_in_its_system(amgt, orc):
    """45 systems of 40 x 35 unknowns and one coarse level: system and coarse
    sizes (1,400 and 360) are multiples of 4, so no block holds two systems,
    but not of 16, so slices of the sliced copies (16 or 32 rows) do.  A NaN in one system's
    right-hand side (whose last slice holds rows of the next one) changes no
    bit of the others' solutions."""
    from amgt_b200.amg import BatchSolver, default_params

    ns, bad = 45, 40
    A, P = orc.laplacian(40, 35, 1), orc.geometric_hierarchy(40, 35, 1)[0]
    n = A.n
    amgt.set_level_policy([0])
    try:
        S = BatchSolver([(to_dev(A), [to_dev(P)])] * ns, default_params(max_coarse_rows=16384))
        lv = S.level(0)
        assert lv["blocks"] >= 65536 and n % 4 == 0 and n % 16 != 0 and P.n % 4 == 0
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
