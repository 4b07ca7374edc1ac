"""The memory that step results live in (ingot_b200.models._Results), without a device."""
import gc

import numpy as np
import pytest

from ingot_b200 import models as M


class Heap:
    """Host memory in the place of pinned memory."""

    def __init__(self, room=1 << 30):
        self.held, self.room = {}, room

    def ingot_model_host_alloc(self, size):
        if size > self.room:
            return None
        block = np.zeros(size, np.uint8)
        self.held[block.ctypes.data] = block
        return block.ctypes.data

    def ingot_model_host_free(self, at):
        del self.held[at]


@pytest.fixture
def heap(monkeypatch):
    h = Heap()
    monkeypatch.setattr(M, "lib", lambda: h)
    return h


def test_a_block_serves_one_result_at_a_time(heap):
    r = M._Results()
    a, b = r.empty(3, 10), r.empty(3, 10)
    assert a.shape == (3, 10) and a.dtype == np.float32 and a.flags.writeable and a.ctypes.data != b.ctypes.data
    a[:], b[:] = 1, 2
    row, at = a[1], a.ctypes.data
    del a
    c = r.empty(3, 10)
    assert c.ctypes.data not in (at, b.ctypes.data) and (row == 1).all()  # a view keeps the block
    del row
    gc.collect()
    assert r.empty(4, 10).ctypes.data == at  # the same size class
    del b, c, r
    gc.collect()
    assert not heap.held


def test_blocks_are_bounded_and_idle_ones_make_room(heap):
    r = M._Results()
    r.BLOCKS, r.BYTES = 4, 400
    held = [r.empty(1, 25) for _ in range(6)]
    assert len(heap.held) == 4 and held[5].base is None and held[5].shape == (1, 25)
    del held
    gc.collect()
    wide = r.empty(1, 100)  # all 400 bytes
    assert wide.base is not None and len(heap.held) == 1 and r.bytes == 400 and r.blocks == 1
    assert r.empty(1, 1).base is None


def test_without_pinned_memory(heap):
    heap.room = 0
    r = M._Results()
    assert r.empty(2, 5).base is None and r.blocks == r.bytes == 0
