"""Page-locked result arrays, with ordinary memory in the place of the library's."""
import ctypes
import gc
import threading

import numpy as np
import pytest

from adam_b200.host_arrays import HostArrays

MB = 1 << 20


class Memory:
    """Stands in for the library: blocks by address, and that each is given back once."""

    def __init__(self):
        self.blocks = {}

    def adam_b200_host_alloc(self, n):
        buf = ctypes.create_string_buffer(n)
        self.blocks[ctypes.addressof(buf)] = buf
        return ctypes.addressof(buf)

    def adam_b200_host_free(self, address):
        del self.blocks[address]

    def locked(self):
        return sum(len(b) for b in self.blocks.values())


@pytest.fixture
def arrays():
    a = HostArrays(Memory())
    yield a
    gc.collect()
    a.close()
    gc.collect()
    assert not a._lib.blocks


def test_arrays_in_reference_cycles():
    """The garbage collector may run, and give arrays back, in the middle of any call."""
    arrays = HostArrays(Memory())

    def work():
        for i in range(3000):
            cycle = [arrays.empty((MB // 8 + 1024 * (i % 40),), np.float64)]
            cycle.append(cycle)
            cycle[0][-1] = i

    old = gc.get_threshold()
    gc.set_threshold(5)
    threads = [threading.Thread(target=work, daemon=True) for _ in range(2)]
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join(timeout=30)
        assert not any(t.is_alive() for t in threads)
    finally:
        gc.set_threshold(*old)
    gc.collect()
    arrays.close()
    assert not arrays._lib.blocks


def test_blocks_are_used_again_and_live_as_long_as_a_view(arrays):
    a = arrays.empty((300, 1000), np.float32)
    a[:] = 1
    view = a[5:7]
    where = a.ctypes.data
    del a
    b = arrays.empty((300, 1000), np.float32)
    b[:] = 2
    assert b.ctypes.data != where and (view == 1).all()
    del view
    assert arrays.empty((299, 1000), np.float32).ctypes.data == where


def test_locked_memory_is_bounded(arrays):
    """Results that a program keeps are ordinary arrays once the bound is reached; unused blocks make room for used ones."""
    arrays.LOCKED_LIMIT = 8 * MB
    kept = [arrays.empty((2 * MB,), np.uint8) for _ in range(10)] + [arrays.empty((MB // 2,), np.uint8)]
    assert arrays._lib.locked() == 8 * MB and arrays._locked == 8 * MB
    for i, a in enumerate(kept):
        a[:] = i
    assert all((a == i).all() for i, a in enumerate(kept))
    del a, kept
    big = arrays.empty((7 * MB,), np.uint8)
    assert big.ctypes.data in arrays._lib.blocks and arrays._lib.locked() <= 8 * MB
    del big


def test_a_library_without_memory_gives_ordinary_arrays(arrays):
    arrays._lib.adam_b200_host_alloc = lambda n: None
    a, b = arrays.empty((MB,), np.float32), arrays.empty((MB // 8,), np.float32)
    a[:], b[:] = 1, 2
    assert arrays._locked == 0 and arrays._small == 0
