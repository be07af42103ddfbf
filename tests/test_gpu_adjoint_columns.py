"""Back-projection and tangent passes by column displacements at the sizes where they can go wrong: columns of one
voxel, a single column, one row of columns, columns longer than a block of the weights (48) and than one batch of the
walk's rows (130 in FP64), limited coupling, the derivative of the pair kernel over several slabs.

Tolerances: the gradient along a direction against a central difference (step 1e-4 relative) of the loss 1e-5, as the
per-voxel differences of the gradient tests; mixed precision against FP64 1e-5, the method's bound; slabs against the
stored kernel the same sums in another order, 1e-11 in FP64 and 1e-5 in mixed precision."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _context(rte, grid, L, prec, mode, thresh=None):
    ctx = rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=thresh)
    rng = np.random.default_rng(sum(grid) + L)
    N = grid[0] * grid[1] * grid[2]
    mua, mus = rng.uniform(0.01, 0.2, N), rng.uniform(0.5, 2.0, N)
    return ctx, mua, mus, rng


@pytest.mark.parametrize("stored", [True, False])
@pytest.mark.parametrize("grid,L,thresh", [((5, 4, 1), 3, None), ((1, 1, 9), 2, None), ((1, 6, 7), 1, None),
                                           ((4, 3, 5), 0, None), ((7, 2, 6), 5, 0.45), ((2, 1, 60), 2, None),
                                           ((1, 2, 130), 1, None), ((3, 4, 6), 7, None)])
def test_gradient_of_odd_grids(rte, grid, L, thresh, stored):
    srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_REL_L2, 600, 1e-13), rte.Detector(nbins=1, faces=63)
    mode = rte.KERNEL_STORE if stored else rte.KERNEL_RECOMPUTE
    ctx, mua, mus, rng = _context(rte, grid, L, rte.PREC_FP64, mode, thresh)
    with ctx:
        ctx.set_medium_voxel(mua * 1.05, mus * 0.97)
        target = ctx.detector_flux(srcs, stop, det)

        def loss(a, s):
            ctx.set_medium_voxel(a, s)
            return float(np.sum((ctx.detector_flux(srcs, stop, det) - target) ** 2))

        ctx.set_medium_voxel(mua, mus)
        _, ga, gs = ctx.gradient(srcs, stop, det, target)
        for _ in range(3):
            da, ds = mua * rng.uniform(0, 1, mua.size), mus * rng.uniform(0, 1, mua.size)
            h = 1e-4
            for d, g, lp, lm in ((da, ga, loss(mua + h * da, mus), loss(mua - h * da, mus)),
                                 (ds, gs, loss(mua, mus + h * ds), loss(mua, mus - h * ds))):
                fd = (lp - lm) / (2 * h)
                assert abs(g @ d - fd) < 1e-5 * np.sum(np.abs(g * d))
    c32, _, _, _ = _context(rte, grid, L, rte.PREC_MIXED, mode, thresh)
    with c32:
        c32.set_medium_voxel(mua, mus)
        _, ga32, gs32 = c32.gradient(srcs, stop, det, target)
    assert rel(ga32, ga) < 1e-5 and rel(gs32, gs) < 1e-5


@pytest.mark.parametrize("n,fp64,tol", [(23, True, 1e-11), (27, False, 1e-5)])
def test_tangent_slabs_equal_the_stored_kernel(rte, n, fp64, tol):
    srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_FIXED, 3, 0.0), rte.Detector(nbins=2, faces=63)
    out = []
    for mode in (rte.KERNEL_STORE, rte.KERNEL_RECOMPUTE):
        ctx, mua, mus, rng = _context(rte, (n, n, n), 1, rte.PREC_FP64 if fp64 else rte.PREC_MIXED, mode)
        with ctx:
            ctx.set_medium_voxel(mua, mus)
            out.append(ctx.fisher(srcs, stop, det, mua * rng.uniform(0, 1, mua.size), 0 * mus, want_J=True)[1])
    assert rel(out[1], out[0]) < tol
