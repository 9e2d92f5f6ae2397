"""A digit-product launch that fails ends the reduced factorization with its
error code: nothing is computed from blocks that were never written."""
import os
import subprocess

from tests.conftest import ROOT


def test_failed_launch_is_reported(tmp_path):
    from hspike_gb300.build import ARCH, OUT, nvcc

    exe = str(tmp_path / "reduced_emu_errors")
    inc = ["-I", os.path.join(ROOT, "hspike_gb300", "csrc"), "-I", os.path.join(ROOT, "include")]
    obj = str(tmp_path / "driver.o")
    subprocess.run(["gcc", "-std=gnu11", "-O1", *inc, "-c", os.path.join(ROOT, "tests", "c", "reduced_emu_errors.c"),
                    "-o", obj], check=True, capture_output=True, text=True)
    subprocess.run([nvcc(), *ARCH, "-cudart", "static", "-Xlinker", "--wrap=cudaGetLastError", obj, os.path.join(OUT, "spike_reduced.o"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
