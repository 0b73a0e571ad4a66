"""GPU parity of the conversion's quad-per-block-row count pass (matrices of
more than 8 entries a row on average) at its limits: block rows of 127 to 129
entries, of 32 and 33 block columns, 8 block rows of more than its 1,024-entry
stage, unsorted and empty rows, diagonal first or not, and a last block row of
1 to 4 rows.  Bit for bit against the oracle."""
import numpy as np
import pytest

from gpu_util import assert_bsr_equal, to_dev

pytestmark = pytest.mark.gpu


def _rows(orc, lens, n, spread, shuffle_every, diag_first, seed):
    rng = np.random.default_rng(seed)
    ia, ja = [0], []
    for r, L in enumerate(lens):
        width = min(n, max(L, spread(r)))
        lo = int(rng.integers(0, n - width + 1))
        cols = lo + np.sort(rng.choice(width, size=L, replace=False))
        if diag_first and L and r < n:
            cols = np.concatenate([[r], cols[cols != r][: L - 1]])
        if shuffle_every and r % shuffle_every == 3:
            cols = rng.permutation(cols)
        ja.extend(int(c) for c in cols)
        ia.append(len(ja))
    return orc.CSR(len(lens), n, np.array(ia, np.int32), np.array(ja, np.int32), rng.standard_normal(len(ja)))


CASES = {
    "127_to_129_entries": lambda orc, m: _rows(orc, ([32, 32, 32, 31] + [32] * 4 + [32, 32, 32, 33]) * 40 + [9] * m,
                                               700, lambda r: 60, 0, False, 1),
    "32_33_block_columns": lambda orc, m: _rows(orc, [30] * 400 + [12] * m, 900, lambda r: 128 + 4 * (r // 4 % 3), 0,
                                                True, 2),
    "stage_overflow": lambda orc, m: _rows(orc, ([40] * 16 + [0, 3] + [30] * 14) * 20 + [25] * m, 800,
                                           lambda r: 100, 0, True, 3),
    "unsorted_among_sorted": lambda orc, m: _rows(orc, [20] * 600 + [17] * m, 640, lambda r: 40, 7, True, 4),
}


@pytest.mark.parametrize("m", [0, 1, 2, 3])
@pytest.mark.parametrize("name", sorted(CASES))
def test_long_rows_bit_exact(amgt, orc, name, m):
    A = CASES[name](orc, m)
    assert_bsr_equal(amgt.Bsr.from_csr(*to_dev(A)), orc.csr2bsr(A))
