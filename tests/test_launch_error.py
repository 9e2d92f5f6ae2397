"""A refused launch is reported once: the next, healthy call does not fail its
own launch check on an error left behind."""
import os
import subprocess

from tests.conftest import ROOT


def test_refused_launch_leaves_no_error(tmp_path):
    from hspike_gb300.build import ARCH, nvcc

    exe = str(tmp_path / "launch_error")
    subprocess.run([nvcc(), *ARCH, "-std=c++17", "-cudart", "static", "-Xlinker", "--wrap=cudaLaunchKernelExC", "-Xlinker",
                    "--wrap=cudaGetLastError", "-I", os.path.join(ROOT, "hspike_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "c", "launch_error.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
