"""Results of a session: arrays on recycled page-locked blocks, ids checked as one array."""
import ctypes as C
import gc
import os

import numpy as np
import pytest

from tnsr_b200 import nn, session


class _Memory:
    """Stands in for the calls that lock and unlock pages."""

    def __init__(self):
        self.live = {}

    def tnsr_b200_host_register(self, address, size):
        self.live[address] = size
        return 0

    def tnsr_b200_host_unregister(self, address):
        del self.live[address]


def _copy(address, floats, value):
    """What the device's copy engine does: fill the page-locked address."""
    np.frombuffer((C.c_float * floats).from_address(address), dtype=np.float32)[:] = value


def test_result_blocks_are_bounded_reused_and_given_back(monkeypatch):
    memory, n = _Memory(), 1 << 18
    monkeypatch.setattr(session, "lib", lambda: memory)
    assert session._ResultBlocks(n - 1).array(n - 1)[0].flags.owndata and not memory.live       # small results are ordinary arrays
    blocks = session._ResultBlocks(n)
    assert len(memory.live) == 2 and blocks.array(n + 1)[0].flags.owndata
    (a, first), (b, second), (c, third) = (blocks.array(n) for _ in range(3))
    assert not np.shares_memory(a, b) and not a.flags.owndata and c.flags.owndata and c.ctypes.data == third
    for array, address in ((a, first), (b, second)):           # what is copied there is seen here, and no array lies on locked pages
        assert address in memory.live and not any(at <= array.ctypes.data < at + size for at, size in memory.live.items())
        _copy(address, n, 0.5)
        assert np.all(array == 0.5)
    a[:], view = 1.0, a[5:9].reshape(2, 2)
    at = a.__array_interface__["data"][0]
    del a, array
    gc.collect()
    held = blocks.array(n)[0]
    held[:] = 2.0
    assert held.flags.owndata and np.all(view == 1.0)          # a view keeps its block
    del view
    gc.collect()
    again = blocks.array(n)[0]
    assert again.__array_interface__["data"][0] == at and len(memory.live) == 2
    del again
    gc.collect()
    blocks.close()
    assert not memory.live                                     # unlocked at once, also under an array that is still the caller's
    b[:] = 3.0
    del b
    gc.collect()                                               # nothing is left to unlock when it goes


def test_a_block_whose_array_a_forked_child_may_read_is_not_used_again(monkeypatch):
    memory, n = _Memory(), 1 << 18
    monkeypatch.setattr(session, "lib", lambda: memory)
    blocks = session._ResultBlocks(n)
    array, address = blocks.array(n)
    _copy(address, n, 4.0)
    parent, child = os.pipe()
    go, wait = os.pipe()
    pid = os.fork()
    if pid == 0:
        os.read(go, 1)
        os.write(child, b"y" if np.all(array == 4.0) else b"n")
        os._exit(0)
    del array
    gc.collect()
    for _ in range(4):
        _, address = blocks.array(n)
        if address in memory.live:
            _copy(address, n, 5.0)
    os.write(wait, b"g")
    assert os.read(parent, 1) == b"y"
    os.waitpid(pid, 0)
    blocks.close()


def test_pages_that_cannot_be_locked_are_ordinary_arrays(monkeypatch):
    memory, n = _Memory(), 1 << 18
    monkeypatch.setattr(memory, "tnsr_b200_host_register", lambda address, size: -9, raising=False)
    monkeypatch.setattr(session, "lib", lambda: memory)
    assert session._ResultBlocks(n).array(n)[0].flags.owndata


@pytest.mark.parametrize("tokens", [[0, 5, 4294967295], (1, 2), [np.uint32(3), np.int64(4)], [True, 0]])
def test_whole_numbers_become_an_array(tokens):
    assert nn._unsigned(tokens).tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("tokens", [[-1], [1 << 32], [1.0], np.arange(3), b"ab", ["1"]])
def test_anything_else_is_left_to_the_general_check(tokens):
    assert nn._unsigned(tokens) is None
