"""What the kept host blocks hold: their limits apply as soon as a block comes back, and a small result that a program
keeps holds no more than a small multiple of itself."""
import gc
import threading

import numpy as np

from computeql_gb300 import ops

MB = 1 << 20


def blocks(limit=None, mapped=None):
    b = ops._ResultBlocks()
    b.LIMIT, b.MAPPED = limit or b.LIMIT, mapped or b.MAPPED
    return b


def held(b):
    return sum(t for _, t in b.free)


def test_limits_apply_when_a_block_comes_back():
    b = blocks(limit=5 * MB)
    results = [b.take(4 * MB, np.uint8) for _ in range(4)]
    del results
    gc.collect()
    assert not b.returned and 0 < held(b) <= 5 * MB
    b = blocks(mapped=20 * MB)
    for _ in range(3):
        used = []
        first, second = b.take(16 * MB, np.uint8, used), b.take(16 * MB, np.uint8, used)
        for note in used:
            note(4096)
        del first, second, note
        used.clear()
        gc.collect()
        assert not b.returned and sum(m.nbytes for m, _ in b.free) <= 20 * MB


def test_a_small_result_keeps_no_block():
    b = blocks()
    used = []
    a = b.take(MB, np.uint32, used)
    a[:10] = range(10)
    rows = b.cut(a, 10, used)
    del a
    used.clear()
    gc.collect()
    assert rows.base is None and rows.tolist() == list(range(10)) and len(b.free) == 1
    # a large one is a view, as long as it is not little of what the block holds
    used = []
    a = b.take(16 * MB, np.uint32, used)
    a[:] = 3
    whole = b.cut(a, 16 * MB, used)
    assert whole.base is not None and np.shares_memory(whole, a)
    del a, whole
    used.clear()
    gc.collect()
    assert held(b) >= 64 * MB
    used = []
    a = b.take(16 * MB, np.uint32, used)      # the touched block again
    part = b.cut(a, MB, used)
    assert part.base is None and len(part) == MB and np.all(part == 3)
    other = b.cut(a, 4 * MB, used)
    assert np.shares_memory(other, a)


def test_a_block_that_holds_more_is_not_taken_for_a_small_result():
    b = blocks()
    a = b.take(64 * MB, np.uint8)
    at = a.ctypes.data
    del a
    gc.collect()
    assert b.take(2 * MB, np.uint8).ctypes.data != at
    assert b.take(32 * MB, np.uint8).ctypes.data == at


def test_a_block_counts_what_its_results_could_touch():
    b = blocks(limit=8 * MB)
    used = []
    a = b.take(64 * MB, np.uint8, used)
    used[0](4096)
    del a
    used.clear()
    gc.collect()
    c = b.take(2 * MB, np.uint8)              # 2 of its 64 MB
    assert not b.free
    del c
    gc.collect()
    assert [t for _, t in b.free] == [2 * MB]


def test_a_return_that_meets_the_lock_is_sorted_in_later():
    b = blocks(limit=5 * MB)
    a = [b.take(4 * MB, np.uint8) for _ in range(3)]
    with b.lock:                              # a destructor never waits for it, whichever thread runs it
        del a
        gc.collect()
    b._settle()
    assert not b.returned and held(b) <= 5 * MB


def test_threads_leave_the_blocks_within_their_limit():
    b = blocks(limit=6 * MB)
    wrong = []

    def work(mark):
        for i in range(60):
            used = []
            a = b.take(MB // 2 + 1000 * (i % 7), np.uint32, used)
            a[::4096] = mark
            c = b.cut(a, 2 * MB // 8, used)
            del a
            if not np.all(c[::4096] == mark):
                wrong.append(mark)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    gc.collect()
    assert not wrong and not b.returned and held(b) <= 6 * MB
