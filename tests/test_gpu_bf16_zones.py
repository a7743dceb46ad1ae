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


@pytest.mark.parametrize("blur", [1, 5, 9])
def test_fewer_kept_candidates_never_find_more(ptk, cuda_device, pair, blur):
    """A tile that has no more candidates near its best one than are kept takes
    them all; one with more (smooth images, a small limit) ranks them.  Either
    way the kept sets of growing limits contain one another and hold the best
    ranked candidate, so the coefficient found grows with the limit, never
    passes the exact one and stays within the weak keep margin (10 %) of it."""
    p = pair["params"]

    def smooth(f):
        for axis in (0, 1):
            f = sum(np.roll(f.astype(np.int64), k, axis) for k in range(-(blur // 2), blur // 2 + 1)) // blur
        return f.astype(np.uint16)

    ref, cur = smooth(pair["ref"]), smooth(pair["cur"])
    out = []
    for method, topk in ((ptk.SEARCH_BF16, 1), (ptk.SEARCH_BF16, 2), (ptk.SEARCH_BF16, 5), (ptk.SEARCH_BF16, 8),
                         (ptk.SEARCH_EXACT, 8)):
        t = ptk.Tracker(p["dimx"], p["dimy"], rescue_level=0, NCC_min=0.01, search_method=method, iraz=100, topk=topk)
        t.set_zone(0, 8, 8, 7, 7, 4, 0.01)
        t.set_grains(pair["rec"])
        t.make_patterns("grain_diameter", 1.0, 1.0)
        t.load_frame(0, ref)
        t.load_frame(1, cur)
        t.search(0)
        out.append(t.get_grains_structs()["NCC"].copy())
        t.close()
    assert np.all(out[0] > 0.0)
    for few, more in zip(out, out[1:]):
        assert np.all(few <= more)
    assert np.all(out[0] >= 0.9 * out[-1])
