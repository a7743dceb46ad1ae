"""The correctly rounded cosine and sine of the plain subpixel objective
(p-tracker_b200/csrc/ptk_crtrig.cuh), compiled for the host: the quick phase
returns what the double-double series returns on every angle that it decides,
it decides nearly all of them, and the results are within an ulp of the C
library's."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    so = tmp_path_factory.mktemp("crtrig") / "libcrtrig_harness.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-fPIC", "-shared",
                    str(HERE / "crtrig_harness.cpp"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.crt_undecided.restype = C.c_long
    return L


def _angles(kind: str, n: int) -> np.ndarray:
    rng = np.random.default_rng(3)
    if kind == "edge":  # the ends of the quick phase's range and of zero's neighbourhood
        a = np.array([0.25, np.nextafter(0.25, 0), np.nextafter(0.25, 1), 5e-324, 1e-300, 1e-160, 1e-20, 2.0 ** -27])
        return np.concatenate([a, -a, 0.25 - rng.uniform(0, 1e-9, n), rng.uniform(0.2, 0.25, n)])
    if kind == "small":
        return rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, -1, n)
    return rng.uniform(-0.25, 0.25, n)


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("kind", ["edge", "small", "range"])
def test_quick_phase_is_the_series(harness, which, kind):
    x = np.ascontiguousarray(_angles(kind, 300000))
    n = len(x)
    a, b = np.zeros(n), np.zeros(n)
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    harness.crt_eval(p(x), C.c_long(n), C.c_int(which), p(a))
    harness.crt_series(p(x), C.c_long(n), C.c_int(which), p(b))
    np.testing.assert_array_equal(a, b)
    lib = np.sin(x) if which else np.cos(x)
    assert (np.abs(a - lib) <= np.spacing(np.abs(lib))).all()
    # an error bound of 2^-62 against half-ulps of 2^-54 leaves one angle in 128 at most
    assert harness.crt_undecided(p(x), C.c_long(n), C.c_int(which)) <= n // 128
