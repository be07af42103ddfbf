"""FP64 solves and mixed solves of small grids do not depend on a timing: the launch tuner's choice of chunks, and with it
the order of the sums, is left to its model there.  Bit for bit against the model's choice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("n,L,prec,mod", [(12, 3, 0, 0.0), (17, 5, 0, 0.0), (19, 1, 0, 0.0), (23, 2, 0, 0.0), (15, 3, 0, 0.7),
                                          (13, 3, 1, 0.0), (15, 1, 1, 0.0)])
def test_chunks_by_the_model(rte, monkeypatch, n, L, prec, mod, mode):
    rng = np.random.default_rng(n)
    mua, mus = rng.uniform(0.005, 0.1, n ** 3), rng.uniform(0.5, 2.0, n ** 3)
    W = rng.standard_normal((n ** 3, (L + 1) ** 2)) + 0j
    out = []
    for tune in ("1", "0"):
        monkeypatch.setenv("RTE_AUTOTUNE", tune)
        with rte.Context(n, n, n, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode) as ctx:
            ctx.set_medium_voxel(mua, mus)
            ctx.set_modulation(mod)
            out.append(ctx.prop_abs(W, 1, 1))
    assert np.array_equal(out[0], out[1])
