"""The register-tiled exact search over zones of every tile shape against the
direct kernel: candidates mapped to lanes by the zone's width and height (1, 2 or
4 warps a column class, inactive lanes, several tiles), and the columns' runs
found by warps (patterns with many runs, repeated offsets, extents around 32
rows).  Both kernels give the same records."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ZONES = [(0, 0, 0, 0), (0, 1, 1, 0), (3, 3, 3, 3), (3, 4, 7, 8), (8, 8, 8, 8), (7, 8, 15, 16), (15, 15, 15, 15), (15, 16, 15, 16),
         (16, 16, 2, 2), (1, 1, 20, 20)]


def _patterns(rng, n):
    out = []
    for i in range(n):
        r = (3, 15, 16, 31, 44)[i % 5]
        y, x = np.mgrid[-r:r + 1, -r:r + 1]
        xy = np.stack([x.ravel(), y.ravel()], 1)[(x * x + y * y <= r * r).ravel()]
        if i % 3 == 1:   # every second row and a few holes: many runs a column
            xy = xy[(xy[:, 1] % 2 == 0) | (rng.random(len(xy)) < 0.1)]
        if i % 3 == 2:   # repeated offsets
            xy = np.concatenate([xy, xy[: len(xy) // 3]])
        out.append(xy)
    return out


@pytest.mark.parametrize("zone", ZONES)
def test_tiled_equals_direct(ptk, cuda_device, zone):
    rng = np.random.default_rng(3)
    ref = rng.integers(0, 65536, (420, 460)).astype(np.uint16)
    cur = np.roll(ref, (2, -1), (0, 1))
    n = 15
    rec = np.zeros((n, 13))
    rec[:, 0] = rng.integers(100, 360, n)
    rec[:, 1] = rng.integers(100, 320, n)
    rec[0, :2] = 30, 200  # leaves the frame for the larger zones
    pats = _patterns(rng, n)
    out = []
    for method in (ptk.SEARCH_EXACT, 2):  # 2: PTK_SEARCH_EXACT_DIRECT
        t = ptk.Tracker(460, 420, rescue_level=0, search_method=method, iraz=100)
        t.set_zone(0, *zone, 2, 0.02)
        t.set_grains(rec)
        t.set_patterns(pats)
        t.load_frame(0, ref)
        t.load_frame(1, cur)
        t.search(0)
        out.append((t.get_grains(), t.status()))
        t.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("r", [32, 50, 51, 59, 60, 61])
def test_extents_and_flat_windows(ptk, cuda_device, r):
    """Extents around 64 rows, around the two patch pitches and up to the largest
    that is tiled, with points beyond those a thread holds, holes and repeated
    offsets; windows of no variance (a coefficient of no value) and of little."""
    rng = np.random.default_rng(r)
    ref = rng.integers(0, 65536, (420, 460)).astype(np.uint16)
    cur = np.roll(ref, (1, -2), (0, 1))
    cur[:, 230:] = 777
    cur[200:, 230:] += (rng.random((220, 230)) < 0.001).astype(np.uint16)
    n = 8
    rec = np.zeros((n, 13))
    rec[:, 0] = rng.integers(100, 360, n)
    rec[:, 1] = rng.integers(100, 320, n)
    rec[0, :2], rec[1, :2] = (345, 100), (345, 310)
    y, x = np.mgrid[-r:r + 1, -r:r + 1]
    disc = np.stack([x.ravel(), y.ravel()], 1)[(x * x + y * y <= r * r).ravel()]
    pats = [disc[rng.random(len(disc)) < (1.0, 0.9, 0.5, 0.02)[i % 4]] for i in range(n)]
    pats[4] = np.concatenate([pats[4], pats[4][:500]])
    out = []
    for method in (ptk.SEARCH_EXACT, 2):  # 2: PTK_SEARCH_EXACT_DIRECT
        t = ptk.Tracker(460, 420, rescue_level=0, search_method=method, iraz=100)
        t.set_zone(0, 5, 6, 4, 6, 2, 0.02)
        t.set_grains(rec)
        t.set_patterns(pats)
        t.load_frame(0, ref)
        t.load_frame(1, cur)
        t.search(0)
        out.append((t.get_grains(), t.status()))
        t.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
