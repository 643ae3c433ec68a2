"""The FD apply takes its pointers from the tensors of the object it is called on: a deep
copy uses its own, and threads that build the device data at the same time never leave a
call with the pointers of a dropped copy. (CPU tensors, FP32 so that the data are copies, and a fake native call.)"""
import copy
import threading

import numpy as np
import pytest
import torch

from igaops_b200 import fastdiag
from igaops_b200.fastdiag import SingleFD
from tests._problems import rules


@pytest.fixture
def calls(monkeypatch):
    """Records (factor pointers, 1 / Lambda pointer) of every native apply."""
    seen = []

    def fake(dtype, ndim, n, lo, m, U, inv, *rest):
        seen.append(([U[d] for d in range(ndim)], inv))
        return 0

    monkeypatch.setattr(fastdiag, "require_cuda", lambda: torch.device("cpu"))
    monkeypatch.setattr(fastdiag, "stream_handle", lambda: 0)
    monkeypatch.setattr(fastdiag._lib.LIB, "iga_fd_apply", fake)
    return seen


def _fd():
    fd = SingleFD("spatial")
    fd.compute_space_eigendecomposition(rules(3, 2, 4), np.ones((1, 3, 2), dtype=bool))
    fd.update_space_eigenvalues([0.0, 1.0])
    return fd.space_preconditioner


def _apply(sp, calls):
    n = int(np.prod(list(sp.nonzeros_by_dir.values())))
    x = torch.zeros(n, dtype=torch.float32)
    sp.apply_device(x, torch.empty_like(x))
    U, inv = sp.device_data(torch.float32)[0]
    assert calls[-1] == ([u.data_ptr() for u in U], inv.data_ptr())


def test_deep_copy_uses_its_own_tensors(calls):
    sp = _fd()
    _apply(sp, calls)
    twin = copy.deepcopy(sp)
    _apply(twin, calls)
    assert calls[0][1] != calls[1][1] and not set(calls[0][0]) & set(calls[1][0])
    del sp
    _apply(twin, calls)


def test_threads_that_build_the_data_together(calls):
    """Two threads form the device data at once; the first one is held after its first
    store until the second is through."""
    sp = _fd()
    stored, second_done = threading.Event(), threading.Event()

    class Held(dict):
        def __setitem__(self, key, value):
            super().__setitem__(key, value)
            if threading.current_thread().name == "first" and not stored.is_set():
                stored.set()
                second_done.wait(30)

        def get(self, key, default=None):  # the second thread looked before the store
            if threading.current_thread().name == "second":
                return default
            return super().get(key, default)

    sp._dev = Held()
    threads = [threading.Thread(target=lambda: sp.device_data(torch.float32), name=name)
               for name in ("first", "second")]
    threads[0].start()
    assert stored.wait(30)
    threads[1].start()
    threads[1].join(30)
    second_done.set()
    threads[0].join(30)
    _apply(sp, calls)


def test_data_dropped_while_a_call_is_prepared(calls, monkeypatch):
    """Another thread that changes the correctors between a call's look-ups."""
    sp = _fd()
    build = sp.device_data

    def build_then_clear(dtype):
        hit = build(dtype)
        sp._dev.clear()
        return hit

    monkeypatch.setattr(sp, "device_data", build_then_clear)
    n = int(np.prod(list(sp.nonzeros_by_dir.values())))
    x = torch.zeros(n, dtype=torch.float32)
    sp.apply_device(x, torch.empty_like(x))
    assert len(calls) == 1
