"""Sums of digit products against exact sums.

What the digits leave out adds up over the terms: the pairs of digits that are
not formed stay below 7.03 * 2^14 * 2^48 per term, the digits below the last one
below 2 * 2 * 2^62 (one unit of 2^-61 of a scale against a value of up to twice the other
scale, on either side), all in units of 2^-122 of the two scales' product.  The
worst inputs are correlated ones -- constant rows and columns, every digit near
its extreme, one sign -- with a sum near the guard's edge."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from hspike_gb300.build import ARCH, nvcc

    so = str(tmp_path_factory.mktemp("slices") / "libslices.so")
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "hspike_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "slices_check.cu"), "-o", so],
                   check=True, capture_output=True, text=True)
    return C.CDLL(so)


def digits(bs, e):
    """the double of exponent e whose byte digits below the leading one are bs (-128 .. 127)"""
    m = 3 << 60
    for i, b in enumerate(bs):
        m += b << (8 * (6 - i))
    return float(Fraction(m) * Fraction(2) ** (e - 61))


def check(lib, a, b):
    K = a.shape[1]
    out, mag = np.zeros((16, 8)), np.zeros((16, 8), np.float32)
    p = [np.ascontiguousarray(v).ctypes.data_as(C.c_void_p) for v in (a, b, out, mag)]
    assert lib.slices_check(p[0], p[1], K, out.ctypes.data_as(C.c_void_p), mag.ctypes.data_as(C.c_void_p)) == 0
    ra = [2.0 ** np.floor(np.log2(np.abs(r).max())) for r in a]
    cb = [2.0 ** np.floor(np.log2(np.abs(c).max())) for c in b.T]
    left = Fraction(K) * (Fraction(703, 100) * 2 ** 62 + 4 * 2 ** 62) / Fraction(2) ** 122
    sums = {}
    for r in range(16):
        for c in range(8):
            key = (a[r].tobytes(), b[:, c].tobytes())
            if key not in sums:
                terms = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a[r], b[:, c])]
                sums[key] = sum(terms), sum(abs(t) for t in terms)
            exact, total = sums[key]
            scale = Fraction(ra[r]) * Fraction(cb[c])
            err = abs(Fraction(float(out[r, c])) - exact)
            assert err <= left * scale + abs(exact) / 2 ** 53, (r, c, float(err / scale))
            # the guard's magnitude never overstates the sum of the terms' magnitudes
            assert Fraction(float(mag[r, c])) * scale <= total


@pytest.mark.parametrize("K", [16, 64, 272])
@pytest.mark.parametrize("pattern", [(-128,) * 7, (127,) * 7, (-128, 127) * 3 + (-128,), (0, 0, 0, 0, -128, -128, -128)])
def test_correlated_digits(lib, K, pattern):
    x = digits(pattern, 0)
    for small in (0, 6, 8, 14):  # every value but the one that sets the scale lies 2^-small below it
        a = np.full((16, K), x * 2.0 ** -small)
        b = np.full((K, 8), x)
        a[:, 0] = x
        b[0, :] = 0.0  # the large value meets nothing
        check(lib, a, b)
        check(lib, a, -b)


@pytest.mark.parametrize("K", [16, 64, 128, 272])
def test_random_values(lib, K):
    rng = np.random.default_rng(K)
    a = rng.uniform(-1, 1, (16, K)) * 2.0 ** rng.integers(-12, 1, (16, K)) * 2.0 ** rng.integers(-40, 40, (16, 1))
    b = rng.uniform(-1, 1, (K, 8)) * 2.0 ** rng.integers(-70, 1, (K, 8)) * 2.0 ** rng.integers(-40, 40, (1, 8))
    check(lib, a, b)
    check(lib, np.abs(a), np.abs(b))
