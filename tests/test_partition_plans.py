"""Requested partition counts: split inside by default, exactly p on request,
and exactly p as well where the pieces do not fit the device's memory; and what
any plan holds against the estimate that requests are admitted by."""
import os
import subprocess

from tests.conftest import ROOT


def test_requested_partition_counts(tmp_path):
    exe = str(tmp_path / "partition_plans")
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-no-pie", "-pthread", "-I", os.path.join(ROOT, "hspike_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "c", "partition_plans.c"), "-o", exe,
                    "-Wl,--unresolved-symbols=ignore-all", "-lm"], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
