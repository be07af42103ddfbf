"""The ctypes binding hands every status to its check with the call's name (no GPU, no library)."""
import numpy as np
import pytest

from doi_b200 import rte


def test_split_tissue_table_checks_its_status():
    seen = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: seen.append(name) or 4

        def rte_last_error(self, h):
            return b"refused"

    ctx = rte.Context.__new__(rte.Context)
    ctx.lib, ctx.h = Lib(), 0
    t = np.array([0.01, 0.1])
    with pytest.raises(rte.RteError, match="rte_set_medium_tissue_split failed"):
        ctx.set_medium_tissue_split(np.zeros(4, np.uint8), t, t, t, t)
    assert "rte_set_medium_tissue_split" in seen
    ctx.h = None
