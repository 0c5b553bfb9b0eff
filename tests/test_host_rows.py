"""The host memory that steps' logits arrive in: kept within its limit, given back by the arrays, whole after its owner is closed."""
from __future__ import annotations

import ctypes as C
import gc
import mmap
import os
import threading

import numpy as np
import pytest

from liyab_b200.engine import _HostRows

PIECE = 65536


class FakeLib:
    """Buffers of ordinary memory, counted; `refuse` stands for an allocation that fails."""

    def __init__(self):
        self.live, self.made, self.refuse = {}, 0, False

    def lb_host_buffer_create(self, device, size, out):
        if self.refuse:
            return 8
        memory = (C.c_char * size)()
        self.live[C.addressof(memory)] = memory
        self.made += 1
        out._obj.value = C.addressof(memory)
        return 0

    def lb_host_buffer_destroy(self, address):
        del self.live[address]


@pytest.fixture
def lib():
    return FakeLib()


def test_buffers_come_back_with_the_last_view(lib):
    rows = _HostRows(limit=4 * PIECE, lib=lib)
    a = rows.array(3, 100)
    a[:] = np.arange(300).reshape(3, 100)
    view = a[1:, ::2]
    del a
    b = rows.array(3, 100)
    assert lib.made == 2 and b.ctypes.data not in (view.ctypes.data, view.base.ctypes.data)
    b[:] = -1.0
    assert (view == np.arange(300).reshape(3, 100)[1:, ::2]).all()
    del view, b
    gc.collect()
    for _ in range(5):
        c = rows.array(3, 100)
        del c
    assert lib.made == 2


def test_limit_and_refusals_give_ordinary_arrays(lib):
    rows = _HostRows(limit=2 * PIECE, lib=lib)
    held = [rows.array(1, PIECE // 4) for _ in range(4)]
    assert lib.made == 2 and all(a.shape == (1, PIECE // 4) and a.flags.writeable for a in held)
    del held
    big = rows.array(2, PIECE // 4)                  # two free buffers make room for one of twice their size
    assert lib.made == 3 and len(lib.live) == 1
    del big
    lib.refuse = True
    assert rows.array(1, 10).shape == (1, 10) and len(lib.live) == 1


def test_arrays_outlive_their_owner(lib):
    rows = _HostRows(limit=4 * PIECE, lib=lib)
    a, b = rows.array(1, 10), rows.array(1, 10)
    a[:] = 3.0
    del b
    rows.close()
    assert len(lib.live) == 1 and (a == 3.0).all()
    assert rows.array(1, 10).shape == (1, 10) and len(lib.live) == 1
    del a
    gc.collect()
    assert not lib.live


def test_threads_never_share_a_buffer(lib):
    rows, wrong = _HostRows(limit=64 * PIECE, lib=lib), []

    def work(k):
        for i in range(200):
            a = rows.array(1, 50)
            a[:] = k
            if (a != k).any():
                wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong and len(lib.live) <= 9


def test_a_request_past_the_limit_leaves_the_buffers(lib):
    rows = _HostRows(limit=4 * PIECE, lib=lib)
    a = rows.array(1, PIECE // 4)
    del a
    for _ in range(3):
        assert rows.array(8, PIECE // 4).shape == (8, PIECE // 4) and len(lib.live) == 1
        rows.array(1, PIECE // 4)
    assert lib.made == 1


def test_sizes_that_do_not_fit_beside_one_another_give_way_seldom(lib):
    rows = _HostRows(limit=4 * PIECE, lib=lib)
    for _ in range(200):
        rows.array(4, PIECE // 4)
        rows.array(1, PIECE // 4)
    assert lib.made <= 2 + 400 // rows.REST


def test_a_caller_who_keeps_its_arrays_soon_gets_ordinary_ones(lib):
    rows = _HostRows(limit=64 * PIECE, lib=lib)
    kept = [rows.array(1, 10) for _ in range(50)]
    assert lib.made == rows.FIRST
    kept[3] = None
    kept.append(rows.array(1, 10))
    assert lib.made == rows.FIRST
    del kept
    for _ in range(20):
        rows.array(1, 10)
    assert lib.made == rows.FIRST


def test_a_caller_who_uses_many_at_a_time_soon_has_buffers_for_all(lib):
    rows = _HostRows(limit=64 * PIECE, lib=lib)
    made = []
    for _ in range(5):
        session = [rows.array(1, 10) for _ in range(17)]
        made.append(lib.made)
        del session
    assert made == [8, 16, 17, 17, 17]


class SharedLib(FakeLib):
    """Buffers that a forked child shares with its parent, as the real ones are."""

    def lb_host_buffer_create(self, device, size, out):
        pages = mmap.mmap(-1, size)
        memory = (C.c_char * size).from_buffer(pages)
        self.live[C.addressof(memory)] = memory
        self.made += 1
        out._obj.value = C.addressof(memory)
        return 0


def test_a_forked_child_keeps_what_it_was_handed():
    lib = SharedLib()
    rows = _HostRows(limit=8 * PIECE, lib=lib)
    a = rows.array(1, 10)
    a[:] = 3.0
    ready, told = os.pipe()
    child = os.fork()
    if child == 0:
        os.read(ready, 1)
        good = (a == 3.0).all() and rows.array(1, 10).shape == (1, 10) and lib.made == 1
        del a
        os._exit(0 if good else 1)
    del a
    gc.collect()
    for _ in range(5):
        b = rows.array(1, 10)
        b[:] = 7.0
        del b
    os.write(told, b"x")
    assert os.waitpid(child, 0)[1] == 0 and lib.made == 2 and len(lib.live) == 1
