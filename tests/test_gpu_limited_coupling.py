"""Coupling over a short distance (prop_thresh): rows of columns that couple with none of a CTA's destinations are left out,
in the pair kernel and in its application.  Against the FP64 oracle, over stored and recomputed kernels, thresholds below
one voxel to beyond the grid, column groups that span several rows, several slabs, the gradient's use of the kernel.

Tolerances: FP64 1e-11 relative L2, mixed precision 1e-5, as the operator's tests; slabs the same sums in another order."""
import numpy as np
import pytest

from conftest import real_to_complex, rel

pytestmark = pytest.mark.gpu


def _medium(N, seed=3):
    t = np.random.default_rng(seed).integers(0, 4, N)
    return np.array([0.01, 0.05, 0.2, 0.1])[t], np.array([1.0, 2.0, 0.5, 1.3])[t]


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("prec,tol", [(0, 1e-11), (1, 1e-5)])
@pytest.mark.parametrize("grid,L", [((5, 14, 6), 3), ((2, 23, 9), 6), ((1, 40, 5), 2), ((9, 30, 1), 1)])
@pytest.mark.parametrize("thresh", [0.05, 0.25, 0.55, 9.0])
def test_operator(rte, oracle, grid, L, thresh, prec, tol, mode):
    N, C = grid[0] * grid[1] * grid[2], (L + 1) ** 2
    mua, mus = _medium(N)
    W = real_to_complex(np.random.default_rng(N).standard_normal((N, C)), L)
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=thresh) as ctx:
        p = oracle.params(*grid, 0.1, 0.1, 0.1, L, 0.8, 1.0, ctx.cfg.prop_thresh, mode=rte.MODEL_EXACT, ssv=1,
                          x_min=ctx.cfg.x_min, y_min=ctx.cfg.y_min, z_min=ctx.cfg.z_min)
        ctx.set_medium_voxel(mua, mus)
        got = ctx.prop_abs(W, 1, 1)
    assert rel(got, oracle.apply(p, mua, mus, W, 1, 1)) < tol


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 2e-6)])
def test_slabs_and_gradient(rte, prec, tol):
    """23^3 FP64 and 27^3 mixed take several slabs when recomputed; the gradient reads the stored kernel or walks."""
    n = (23, 27)[prec]
    mua, mus = _medium(n ** 3)
    W = real_to_complex(np.random.default_rng(n).standard_normal((n ** 3, 4)), 1)
    srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_FIXED, 4), rte.Detector(nbins=2, faces=63)
    out = []
    for mode in (rte.KERNEL_STORE, rte.KERNEL_RECOMPUTE):
        with rte.Context(n, n, n, dx=0.1, nL=1, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=0.35) as ctx:
            ctx.set_medium_voxel(mua * 1.05, mus)
            target = ctx.detector_flux(srcs, stop, det)
            ctx.set_medium_voxel(mua, mus)
            out.append((ctx.prop_abs(W, 1, 0),) + tuple(ctx.gradient(srcs, stop, det, target)[1:]))
    assert rel(out[1][0], out[0][0]) < tol
    # the loss' gradient follows the difference of two fluxes 5 % apart: its errors are some 20 to 40 times theirs
    assert rel(out[1][1], out[0][1]) < 50 * tol and rel(out[1][2], out[0][2]) < 50 * tol
