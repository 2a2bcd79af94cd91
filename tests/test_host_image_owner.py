"""Whether a read-back's host memory is free hangs on its arrays alone, not on
how many references the interpreter counts for a local name (it may borrow
them), and two threads never get the same memory."""

import sys
import threading

import numpy as np
import pytest

from kittlespt_gb300.renderer import Renderer


def _renderer():
    r = Renderer.__new__(Renderer)
    r._host = []
    return r


@pytest.mark.parametrize("borrowed", [0, 1, 2])
def test_with_references_borrowed(monkeypatch, borrowed):
    count = sys.getrefcount
    monkeypatch.setattr(sys, "getrefcount", lambda o: count(o) - 1 - borrowed)   # 1: this function's argument
    r = _renderer()
    held = [r._host_image((4, 6, 4))]
    held[0][...] = 1.0
    views = [held[0][1:3], held[0].reshape(-1)]
    held.append(r._host_image((4, 6, 4)))
    held[1][...] = 2.0
    del held[0]
    for k in range(6):
        r._host_image((4, 6, 4))[...] = 3.0 + k
    assert all((v == 1.0).all() for v in views) and (held[0] == 2.0).all()


def test_threads_get_memory_of_their_own():
    r = _renderer()
    wrong = []

    def work(k):
        for _ in range(300):
            a = r._host_image((8, 8, 4))
            a[...] = k
            if not (a == k).all():
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not wrong and len(r._host) == 2
