"""The tensor-core search over zones of every tile shape: the MMAs cover only the
y offsets and x shifts of 8 columns that the zone needs, so widths around the
multiples of 8 and heights around the even numbers, one pixel, one tile and
just above, with unequal sides and footprints of one and several strips.  The
integer stage equals the exact search's at the default acceptance threshold
(below it a grain is searched again exactly; above it the ranking holds for
matches, which a lower threshold would not ask for)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ZONES = [(0, 0, 0, 0), (0, 1, 1, 1), (3, 4, 0, 1), (4, 4, 2, 2), (7, 8, 5, 6), (8, 8, 7, 7), (11, 12, 15, 15),
         (12, 12, 15, 16), (15, 16, 15, 16), (16, 16, 3, 3), (3, 3, 16, 17)]


@pytest.fixture(scope="module")
def pair(wl):
    p = dict(wl.PRESETS["small16"], dimx=768, dimy=640, n=40, mix=[(0.5, 3.0, 12.0), (0.5, 30.0, 44.0)], zone=20, disp=3.0)
    return wl.make_pair(p, seed=9)


@pytest.mark.parametrize("zone", ZONES)
def test_integer_stage_equals_the_exact_search(ptk, cuda_device, pair, zone):
    p = pair["params"]
    out = []
    for method in (ptk.SEARCH_EXACT, ptk.SEARCH_BF16):
        t = ptk.Tracker(p["dimx"], p["dimy"], rescue_level=0, NCC_min=0.7, search_method=method, iraz=100)
        t.set_zone(0, *zone, 4, 0.01)
        t.set_grains(pair["rec"])
        t.make_patterns("grain_diameter", 1.0, 1.0)
        t.load_frame(0, pair["ref"])
        t.load_frame(1, pair["cur"])
        t.search(0)
        out.append(t.get_grains())
        t.close()
    np.testing.assert_array_equal(out[0], out[1])
