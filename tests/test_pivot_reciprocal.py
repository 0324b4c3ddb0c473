"""The reciprocals of the factorisation's pivots (csrc/pivot.h), compiled on their own with the host compiler: against exact
ones over mantissas and over the whole range of pivots that are taken, and what is refused at its ends.  No GPU."""
import ctypes as C
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "groundtruth_gb300" / "csrc"
SHIM = """
#include "pivot.h"
extern "C" double recip(double d) { return gt::recip64(d); }
extern "C" int pivot(double* v) { return gt::pivot_recip(v[0], v[1]); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cc = shutil.which("g++")
    if not cc:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("pivot")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cc, "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(d / "shim.so")],
                   check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.recip.restype, lib.recip.argtypes = C.c_double, [C.c_double]
    return lib


def test_reciprocal(lib):
    # the last step's rounding, half an ulp of a value in (1/2, 1], and what two steps from FP32 leave
    bound = Fraction(101, 100) / 2 ** 53
    rng = np.random.default_rng(1)
    mant = np.concatenate([1 + rng.random(20000), [1.0, np.nextafter(1, 2), np.nextafter(2, 1), 4 / 3, 1.5]])
    expo = np.concatenate([rng.integers(-1022, 1022, len(mant) - 4), [-1022, -1021, 1020, 1021]])
    for m, e in zip(mant.tolist(), expo.tolist()):
        d = float(np.ldexp(m, e))
        assert abs(Fraction(lib.recip(d)) * Fraction(d) - 1) <= bound, (m, e)


def _recip(lib, re, im):
    v = (C.c_double * 2)(re, im)
    return lib.pivot(v), v[0], v[1]


def test_pivots_of_every_size(lib):
    # the square's two roundings, the reciprocal's and the product's: 2 x 2^-53 + 1.01 x 2^-53 + 2^-53
    bound = Fraction(5) / 2 ** 53
    rng = np.random.default_rng(2)
    size = np.concatenate([10 ** rng.uniform(-149.9, 154, 4000), 10 ** rng.uniform(153.5, 154.127, 4000)])
    ang = rng.uniform(0, 2 * np.pi, len(size))
    for s, a in zip(size, ang):
        re, im = float(s * np.cos(a)), float(s * np.sin(a))
        ok, x, y = _recip(lib, re, im)
        assert ok
        # |(x + j y) (re + j im) - 1|^2 against the bound's square
        p = Fraction(x) * Fraction(re) - Fraction(y) * Fraction(im) - 1
        q = Fraction(x) * Fraction(im) + Fraction(y) * Fraction(re)
        assert p * p + q * q <= bound * bound, (re, im)


@pytest.mark.parametrize("re,im", [(0.0, 0.0), (1e-150, 0.0), (0.0, -9e-151), (1.35e154, 0.0), (1e154, 1e154),
                                   (float("inf"), 0.0), (0.0, float("nan")), (float("nan"), 1.0)])
def test_what_has_no_reciprocal_is_refused(lib, re, im):
    assert _recip(lib, re, im) == (0, 1e150, 0.0)
