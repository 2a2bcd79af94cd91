"""The read-backs' host images: memory is used again only when no array or
view of it is left, and at most two images are kept per renderer."""

import numpy as np
import pytest

from kittlespt_gb300.renderer import Renderer


def _renderer():
    r = Renderer.__new__(Renderer)
    r._host = []
    return r


@pytest.mark.parametrize("hold", ["array", "slice", "reshaped", "memoryview"])
def test_a_held_image_is_not_overwritten(hold):
    r = _renderer()
    a = r._host_image((4, 6, 4))
    a[...] = 1.0
    kept = {"array": lambda x: x, "slice": lambda x: x[1:3, ::2], "reshaped": lambda x: x.reshape(-1),
            "memoryview": memoryview}[hold](a)
    del a
    for k in range(5):
        r._host_image((4, 6, 4))[...] = 2.0 + k
    assert (np.asarray(kept) == 1.0).all()


def test_memory_is_used_again_and_bounded():
    r = _renderer()
    place = r._host_image((8, 8, 4)).ctypes.data
    assert r._host_image((8, 8, 4)).ctypes.data == place
    held = [r._host_image((8, 8, 4)) for _ in range(6)]
    assert len({h.ctypes.data for h in held}) == 6 and len(r._host) == 2
    b = r._host_image((2, 3, 4))
    assert b.shape == (2, 3, 4) and b.flags["C_CONTIGUOUS"] and b.flags["WRITEABLE"] and len(r._host) == 2
