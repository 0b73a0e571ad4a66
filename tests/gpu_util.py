"""Helpers shared by the GPU parity tests (test infrastructure)."""
import numpy as np
import torch


def to_dev(A):
    """oracle CSR -> (m, n, ia, ja, a) on cuda:0."""
    return (A.m, A.n, torch.from_numpy(A.ia).cuda(), torch.from_numpy(A.ja).cuda(), torch.from_numpy(A.a).cuda())


def bsr_host(B):
    h = B.host()
    return h["bptr"], h["bidx"], h["bmap"], h["bval"]


def assert_bsr_equal(gpu, orc_bsr, values=True):
    bptr, bidx, bmap, bval = bsr_host(gpu)
    np.testing.assert_array_equal(bptr, orc_bsr.bptr)
    np.testing.assert_array_equal(bidx, orc_bsr.bidx)
    np.testing.assert_array_equal(bmap, orc_bsr.bmap)
    if values:
        # bit for bit
        np.testing.assert_array_equal(bval.view(np.uint64), orc_bsr.bval.view(np.uint64))


def random_csr(orc, m, n, row_len, seed, dense_rows=()):
    """Random CSR with the diagonal (when in range) first, then random
    distinct columns; rows listed in dense_rows get dense_rows[r] entries."""
    rng = np.random.default_rng(seed)
    ia, ja = [0], []
    lens = dict(dense_rows) if isinstance(dense_rows, dict) else {}
    for r in range(m):
        L = lens.get(r, int(rng.integers(0, row_len + 1)))
        L = min(L, n)
        cols = rng.choice(n, size=L, replace=False)
        if r < n and L > 0:
            cols = cols[cols != r][: L - 1]
            cols = np.concatenate([[r], cols])
        ja.extend(int(c) for c in cols)
        ia.append(len(ja))
    ja = np.array(ja, np.int32)
    a = rng.standard_normal(len(ja))
    return orc.CSR(m, n, np.array(ia, np.int32), ja, a)


class AllocLog:
    """Context in which the library allocates through torch: logs every
    allocation's bytes (self.sizes, in order) and fails those that
    fail(sizes so far, this one last) asks for.  Blocks are held until the context ends;
    every library object made inside must be freed inside."""

    def __init__(self, amgt, fail=None):
        import ctypes

        self._amgt, self._fail, self._held, self.sizes, self.failed = amgt, fail, {}, [], 0
        alloc_t = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p)
        free_t = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)
        self._cb = alloc_t(self._alloc), free_t(lambda ptr, stream, ctx: None)
        self._ptr = [ctypes.cast(f, ctypes.c_void_p) for f in self._cb]

    def _alloc(self, nbytes, stream, ctx):
        self.sizes.append(nbytes)
        if self._fail and self._fail(self.sizes):
            self.failed += 1
            return None
        t = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        self._held[t.data_ptr()] = t
        return t.data_ptr()

    def __enter__(self):
        torch.cuda.synchronize()
        assert self._amgt.lib().amgt_set_allocator(*self._ptr, None) == 0
        return self

    def __exit__(self, *exc):
        torch.cuda.synchronize()
        assert self._amgt.lib().amgt_set_allocator(None, None, None) == 0
        self._held.clear()


def sliced_steps(A):
    """Steps (of 32 slots) of the sliced copy of an operator with the CSR
    pattern of A, restated on the host: 32 >> t rows a slice, 1 << t lanes a
    row, each slice as long as its longest row."""
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    lens, avg, t = np.diff(A.ia), A.ja.size / A.m, 0
    while t < 3 and (A.m << t) // 32 < 24 * sm and avg >= (4 << t):
        t += 1
    rows = 32 >> t
    lens = np.concatenate([lens, np.zeros(-len(lens) % rows, lens.dtype)]).reshape(-1, rows)
    return int(np.maximum(1, (lens.max(1) + (1 << t) - 1) >> t).sum())
