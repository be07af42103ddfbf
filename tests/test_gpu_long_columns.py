"""Mixed precision at L = 7 in columns of more than 512 voxels, whose angle rows hold FP64 pairs, and at the lengths around
which runs of sources change: against the FP64 method (tolerance 2e-6, FP32 rounding of sums over a few columns), real
and complex mu_t."""
import numpy as np
import pytest

from conftest import real_to_complex, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mod", [0.0, 0.7])
@pytest.mark.parametrize("grid,L", [((1, 1, 512), 7), ((1, 2, 513), 7), ((2, 1, 700), 7), ((1, 1, 430), 7), ((1, 2, 347), 7),
                                    ((1, 1, 900), 6), ((1, 1, 1024), 5), ((1, 1, 1024), 7)])
def test_mixed_matches_fp64(rte, grid, L, mod):
    N, C = grid[0] * grid[1] * grid[2], (L + 1) ** 2
    rng = np.random.default_rng(N)
    mua, mus = rng.uniform(0.001, 0.01, N), rng.uniform(0.05, 0.2, N)
    W = real_to_complex(rng.standard_normal((N, C)), L)
    out = []
    for prec in (rte.PREC_FP64, rte.PREC_MIXED):
        with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=rte.KERNEL_STORE) as ctx:
            ctx.set_medium_voxel(mua, mus)
            ctx.set_modulation(mod)
            out.append([ctx.prop_abs(W, flag, 1) for flag in (1, 0)])
    assert all(rel(b, a) < 2e-6 for a, b in zip(*out))
