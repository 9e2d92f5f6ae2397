"""A chain of 64-row FP64 tiles whose wait for a copy runs out leaves with the
error bit set and only once its other copies have landed: they would write
into the shared memory of whichever block comes next."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


def test_other_copies_land_before_the_block_leaves(tmp_path):
    from hspike_gb300.build import ARCH, nvcc

    so = str(tmp_path / "libemu_leave.so")
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "hspike_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "emu_leave.cu"), "-o", so],
                   check=True, capture_output=True, text=True)
    L = C.CDLL(so)
    v = np.random.default_rng(1).standard_normal(64 * 64)
    got = v.copy()
    err, out = (C.c_uint * 1)(), (C.c_int * 2)()
    assert L.leave_check(got.ctypes.data_as(C.c_void_p), err, out) == 0  # the context survived
    assert err[0] == 8  # SPK_DEV_ERR_TIMEOUT
    assert out[0] == 1 and out[1] == 1
    assert np.array_equal(got, v)
