"""Results of a session: arrays on recycled page-locked blocks, ids checked as one array."""
import gc

import numpy as np
import pytest

from tnsr_b200 import nn, session


class _Memory:
    """Stands in for the allocator of page-locked memory."""

    def __init__(self):
        self.live = {}

    def tnsr_b200_host_alloc(self, size):
        block = np.zeros(size, dtype=np.uint8)
        self.live[block.ctypes.data] = block
        return block.ctypes.data

    def tnsr_b200_host_free(self, address):
        del self.live[address]


def test_result_blocks_are_bounded_reused_and_given_back(monkeypatch):
    memory, n = _Memory(), 1 << 18
    monkeypatch.setattr(session, "lib", lambda: memory)
    assert session._ResultBlocks(n - 1).array(n - 1).flags.owndata and not memory.live       # small results are ordinary arrays
    blocks = session._ResultBlocks(n)
    assert len(memory.live) == 2 and blocks.array(n + 1).flags.owndata
    a, b, c = (blocks.array(n) for _ in range(3))
    assert not np.shares_memory(a, b) and not a.flags.owndata and c.flags.owndata
    a[:], view = 1.0, a[5:9].reshape(2, 2)
    at = a.__array_interface__["data"][0]
    del a
    gc.collect()
    held = blocks.array(n)
    held[:] = 2.0
    assert held.flags.owndata and np.all(view == 1.0)          # a view keeps its block
    del view
    gc.collect()
    again = blocks.array(n)
    assert again.__array_interface__["data"][0] == at and len(memory.live) == 2
    del again
    gc.collect()
    blocks.close()
    assert len(memory.live) == 1
    b[:] = 3.0                                                 # still the caller's
    del b
    gc.collect()
    assert not memory.live


@pytest.mark.parametrize("tokens", [[0, 5, 4294967295], (1, 2), [np.uint32(3), np.int64(4)], [True, 0]])
def test_whole_numbers_become_an_array(tokens):
    assert nn._unsigned(tokens).tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("tokens", [[-1], [1 << 32], [1.0], np.arange(3), b"ab", ["1"]])
def test_anything_else_is_left_to_the_general_check(tokens):
    assert nn._unsigned(tokens) is None
