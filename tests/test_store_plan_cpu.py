"""Launch plans of the pair-kernel precompute, built for the host with g++: no grid may get a layout that the shared
memory of a CTA cannot hold.  Runs on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "doi_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_every_plan_fits(tmp_path):
    exe = str(tmp_path / "store_plan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "store_plan_check.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    fields = out.stdout.split()
    assert int(fields[1]) > 100000 and int(fields[3]) > 1000 and int(fields[5]) == 0, out.stdout
