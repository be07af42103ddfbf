"""oracle/build.sh builds the oracle alone where the reference's sources are not there (no directory, or an empty one)."""
import os
import shutil
import subprocess

import pytest

ORACLE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle")


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
@pytest.mark.parametrize("made", [False, True])
def test_without_the_reference(tmp_path, made):
    for f in ("build.sh", "rte_oracle.cpp"):
        shutil.copy(os.path.join(ORACLE, f), tmp_path)
    ref = tmp_path / "reference"
    if made:
        ref.mkdir()
    r = subprocess.run(["bash", str(tmp_path / "build.sh")], env=dict(os.environ, RTE_REFERENCE_DIR=str(ref)),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert (tmp_path / "liboracle.so").exists()
