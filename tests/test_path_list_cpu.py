"""The closed-form path lists of the kernel precompute and the gradient's walk (doi_b200/csrc/rte_walk.cuh), built for the
host with g++ and compared with a sequential walk: ranks, steps, lengths, the order of ties, displacements up to 1023."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "doi_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_lists_are_the_walks(tmp_path):
    exe = str(tmp_path / "path_list_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "path_list_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    fields = out.stdout.split()
    assert int(fields[1]) > 5000 and int(fields[5]) > 5000 and int(fields[7]) == 0, out.stdout
