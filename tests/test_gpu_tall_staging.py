"""The pair-kernel precompute on grids whose mu_t fits shared memory beside the lists, but not beside the tiles of a tall
z block as well: the operator against the FP64 oracle on sampled destinations, the derivative form against a central
difference.

Tolerances: FP64 1e-11 relative L2 (sums of up to N terms of 1e-16 each), mixed precision 1e-5, the method's bound; the
difference of converged solves (the tangent series is the derivative of the converged solve, not of one cut at a number
of terms) with step h = 1e-4 of the medium is off by h^2 times the ratio of third to first derivatives, some tens at the
optical depths here (below 5): 1e-6."""
import numpy as np
import pytest

from conftest import real_to_complex, rel

pytestmark = pytest.mark.gpu


def _medium(N, seed):
    t = np.random.default_rng(seed).integers(0, 4, N)
    return np.array([0.01, 0.05, 0.2, 0.1])[t], np.array([1.0, 2.0, 0.5, 1.3])[t]


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("grid,prec,tol", [((30, 30, 44), 1, 1e-5), ((28, 28, 48), 1, 1e-5), ((17, 17, 48), 0, 1e-11),
                                           ((20, 20, 42), 0, 1e-11), ((13, 13, 96), 0, 1e-11)])
def test_operator(rte, oracle, grid, prec, tol, mode):
    N, L = grid[0] * grid[1] * grid[2], 1
    mua, mus = _medium(N, 3)
    rng = np.random.default_rng(4)
    W = real_to_complex(rng.standard_normal((N, 4)), L)
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode) as ctx:
        ctx.set_medium_voxel(mua, mus)
        got = ctx.prop_abs(W, 1, 1)
        p = oracle.params(*grid, 0.1, 0.1, 0.1, L, 0.8, 1.0, ctx.cfg.prop_thresh, mode=oracle.MODE_EXACT,
                          x_min=ctx.cfg.x_min, y_min=ctx.cfg.y_min, z_min=ctx.cfg.z_min)
    dests = np.sort(rng.choice(N, 96, replace=False))
    ref = oracle.apply_subset(p, mua, mus, W, dests, 1, 1)
    assert rel(got[dests], ref[dests]) < tol


def test_derivative(rte):
    grid, L, h = (17, 17, 48), 1, 1e-4
    N = grid[0] * grid[1] * grid[2]
    mua, mus = _medium(N, 5)
    d = mua * np.random.default_rng(6).uniform(0, 1, N)
    srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_REL_L2, 600, 1e-13), rte.Detector(nbins=2, faces=63)
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=rte.PREC_FP64) as ctx:
        flux = []
        for s in (h, -h):
            ctx.set_medium_voxel(mua + s * d, mus)
            flux.append(ctx.detector_flux(srcs, stop, det))
        ctx.set_medium_voxel(mua, mus)
        J = ctx.fisher(srcs, stop, det, d, 0 * d, want_J=True)[1]
    assert rel(np.ravel(J), np.ravel((flux[0] - flux[1]) / (2 * h))) < 1e-6
