"""The distortion residual kernel's two forms: threads that hold their pairs'
unit vectors (up to two pairs a thread of the fixed grid, 303,104 in all) and
threads that form them again for every image.  Residuals equal the oracle's bit
for bit and the objective its sum, below, at and above the line."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = 592 * 256


@pytest.mark.parametrize("npairs", [1, GRID - 1, GRID + 1, 2 * GRID, 2 * GRID + 1])
@pytest.mark.parametrize("images", [1, 3])
def test_residuals_on_both_sides(ptk, wl, oracle, cuda_device, npairs, images):
    d = wl.make_disto_case(seed=2, n=790, n_tracked=images)
    pairs = ptk.disto_pairs(d["refx"], d["refy"], 0.0, 1e9)
    assert len(pairs) >= 2 * GRID + 1
    pairs = np.ascontiguousarray(pairs[:npairs])
    f = ptk.DistoFit(d["dimx"], d["dimy"], d["refx"], d["refy"], d["dx"], d["dy"], d["ncc"], 0.7, pairs)
    X = d["X"].copy()
    X[4], X[7], X[10] = 1e-22, 1e-9, 0.02
    v, res = f.residuals(X)
    ov, ores = oracle.disto_objective(X, d["refx"], d["refy"], d["dx"], d["dy"], d["ncc"], 0.7, pairs,
                                      with_residuals=True)
    np.testing.assert_array_equal(res, ores)
    # the same terms added in another order: a relative 2^-53 per addition
    assert abs(v - ov) <= images * npairs * 2.0 ** -53 * ov
    assert f.objective(X) == v
    f.close()


def test_unperturbed_parameters_stay(ptk, wl, cuda_device):
    """Directions of zero length leave their parameters as they are, whichever
    other parameters move."""
    d = wl.make_disto_case(seed=4, n=200, n_tracked=2)
    pairs = ptk.disto_pairs(d["refx"], d["refy"], 0.0, 1000.0)
    X0, step = d["X"].copy(), np.zeros(14)
    X0[2:4], step[2] = 0.0, 1e-10
    f = ptk.DistoFit(d["dimx"], d["dimy"], d["refx"], d["refy"], d["dx"], d["dy"], d["ncc"], 0.7, pairs)
    x, ini, end, _ = f.fit(X0, step)
    assert end < ini and x[2] != 0.0
    keep = np.arange(14) != 2
    np.testing.assert_array_equal(x[keep], X0[keep])
    assert end == f.objective(x) / 2
    f.close()
