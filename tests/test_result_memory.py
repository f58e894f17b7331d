"""The host memory that a context's results lie in: a block is used again only when no array is left in
it, in any order and from any thread, and what waits unused is bounded."""
import gc
import threading

import numpy as np
import pytest

from barnacle_gb300.api import _ResultMemory


def address(a):
    return a.__array_interface__["data"][0]


def test_a_block_comes_back_when_the_last_view_goes():
    m = _ResultMemory()
    a = m.array((300, 400), np.float32)
    assert a.shape == (300, 400) and a.dtype == np.float32 and a.flags.writeable and a.flags.c_contiguous
    at = address(a)
    a[:] = 7
    row = a[123, 5:9]
    del a
    gc.collect()
    b = m.array((300, 400), np.float32)
    assert address(b) != at  # the row still lies there
    b[:] = 1
    assert (row == 7).all()
    del row
    gc.collect()
    assert address(m.array((300, 400), np.float32)) == at


def test_sizes_share_blocks_within_a_factor_of_two():
    m = _ResultMemory()
    at = address(m.array(1 << 20, np.uint8))
    assert address(m.array((1 << 19) - 1, np.uint8)) != at
    assert address(m.array(1 << 19, np.uint8)) == at
    assert address(m.array((1 << 20) + 1, np.uint8)) != at


@pytest.mark.parametrize("shape", [0, 1, (0, 3), (3, 5)])
def test_small_results_are_plain_zeros(shape):
    m = _ResultMemory()
    a = m.array(shape, np.int32)
    assert a.base is None or not m._free
    assert not a.any() and a.shape == np.zeros(shape).shape


def test_unused_memory_is_bounded_and_goes_with_its_owner(monkeypatch):
    m = _ResultMemory()
    monkeypatch.setattr(_ResultMemory, "LIMIT", 10 << 20)
    held = [m.array(3 << 20, np.uint8) for _ in range(8)]
    del held
    gc.collect()
    assert 0 < sum(b.nbytes for b in m._free) <= 10 << 20
    a = m.array(3 << 20, np.uint8)
    del m  # the array outlives its home
    gc.collect()
    a[:] = 5
    assert a.sum() == 5 * a.size


def test_threads_never_share_a_block():
    m = _ResultMemory()
    wrong = []

    def work(k):
        for i in range(200):
            a = m.array(1 << 17, np.uint8)
            a[:] = k
            b = a[::4097].copy()
            if not (b == k).all():
                wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_blocks_written_long_ago_are_let_go():
    m = _ResultMemory()
    a, b = m.array(1 << 20, np.uint8), m.array(1 << 20, np.uint8)
    at = {address(a), address(b)}
    del a, b
    c = m.array(1 << 20, np.uint8, stale=1e9)
    assert address(c) in at and len(m._free) == 1
    del c
    d = m.array(1 << 20, np.uint8, stale=-1)  # both are older than that
    assert not m._free
    del d
    assert len(m._free) == 1
