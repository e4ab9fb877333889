"""Result arrays over kept host blocks: a block is handed out again only when no array over it is left, from any thread,
and the free blocks stay within their limit."""
import gc
import threading

import numpy as np

from computeql_gb300 import ops


def blocks(limit=None):
    b = ops._ResultBlocks()
    if limit:
        b.LIMIT = limit
    return b


def test_a_block_waits_for_its_last_view():
    b = blocks()
    a = b.take(1 << 19, np.uint32)
    a[:] = 7
    at, view = a.ctypes.data, a[100:200].view(np.int32)
    del a
    gc.collect()
    other = b.take(1 << 19, np.uint32)
    assert other.ctypes.data != at
    other[:] = 9
    assert np.all(view == 7)
    del view
    gc.collect()
    again = b.take(1 << 18, np.float64)
    assert again.ctypes.data == at and again.dtype == np.float64 and again.flags.writeable


def test_small_results_and_the_limit():
    b = blocks(limit=5 << 20)
    assert b.take(10, np.uint32).base is None
    held = [b.take(4 << 20, np.uint8) for _ in range(4)]
    del held
    gc.collect()
    b.take(1 << 20, np.uint8)
    assert sum(t for _, t in b.free) <= 5 << 20
    used = []
    big = b.take(64 << 20, np.uint8, used)
    used[0](4096)                       # only the first page was written: the block counts for that
    del big, used
    gc.collect()
    b.take(1 << 20, np.uint8)
    assert any(m.nbytes > 64 << 20 for m, _ in b.free)


def test_threads_never_share_a_block():
    b = blocks()
    wrong = []

    def work(mark):
        for i in range(50):
            a = b.take((1 << 18) + 1000 * (i % 7), np.uint32)
            a[::4096] = mark
            c = a[4096:]
            del a
            if not np.all(c[::4096] == mark):
                wrong.append(mark)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
