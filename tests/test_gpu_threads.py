"""Host threads on one device whose calls size a kernel's shared memory
differently."""
import pytest
import torch

from gpu_util import assert_bsr_equal, to_dev

pytestmark = pytest.mark.gpu


def _in_threads(works):
    """Runs each work(stream) in a host thread of its own, on its own
    stream; returns what they raised."""
    import threading

    errors, gate = [], threading.Barrier(len(works))

    def body(work):
        try:
            torch.cuda.set_device(0)
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                gate.wait(60)
                work(st)
                st.synchronize()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=body, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_host_threads_with_wide_products_of_different_sizes(amgt, orc):
    """Products of wide C rows (more than 48 blocks on average) whose longest
    rows, 75 and 65 blocks, take different amounts of shared memory: threads
    multiplying both at once all succeed, with the same values."""
    ops = [amgt.Bsr.from_csr(*to_dev(orc.box(nx, 40, 24))) for nx in (40, 41)]
    want = [amgt.spgemm(G, G, want_csr=False)[0] for G in ops]
    assert [C.s.max_blc_per_row for C in want] == [75, 65]
    torch.cuda.synchronize()

    def work(k):
        def run(st):
            for _ in range(1500):
                C, _ = amgt.spgemm(ops[k], ops[k], want_csr=False, stream=st)
            assert torch.equal(C.val(), want[k].val())

        return run

    assert _in_threads([work(i % 2) for i in range(4)]) == []


def test_host_threads_converting_long_rows_of_different_lengths(amgt, orc):
    """Conversions of matrices of 24.4 and 25.4 entries a row, whose fill
    passes stage different amounts of shared memory (both above 48 KB):
    threads converting both at once all succeed, bit for bit."""
    mats = [orc.box(20, 20, 20), orc.box(40, 40, 24)]
    want = [orc.csr2bsr(A) for A in mats]
    devs = [to_dev(A) for A in mats]
    torch.cuda.synchronize()

    def work(k):
        def run(st):
            for _ in range(1500):
                G = amgt.Bsr.from_csr(*devs[k], stream=st)
            assert_bsr_equal(G, want[k])

        return run

    assert _in_threads([work(i % 2) for i in range(8)]) == []
