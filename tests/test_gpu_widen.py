"""8-bit frames as the context holds them: the values unchanged, for widths below,
at and around the sixteen pixels a thread widens and the block's share, and rows
with a stride of their own."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [4, 15, 16, 17, 63, 64, 65, 511, 512, 2047, 2048, 2064, 4100])
@pytest.mark.parametrize("slot", [0, 1])
def test_widened_frame(ptk, cuda_device, w, slot):
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (9, w + 5)).astype(np.uint8)
    t = ptk.Tracker(w, 9)
    t.load_frame(slot, np.ascontiguousarray(img[:, :w]))
    np.testing.assert_array_equal(t.read_frame(slot), img[:, :w])
    rc = t._L.ptk_load_frame(t.h, slot, C.c_void_p(img.ctypes.data + 3), w, 9, 1, img.strides[0])
    assert rc == 0
    np.testing.assert_array_equal(t.read_frame(slot), img[:, 3:w + 3])
    t.close()
