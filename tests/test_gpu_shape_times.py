"""Times of solves whose grids are far from a cube, against a cube of about as many voxels.  Bounds are wide: several times
what was measured, and several times below what the shapes took when a part of the work ran on one CTA."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ms(f, reps=3):
    f()
    t = []
    for _ in range(reps):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t) * 1e3


def _medium(grid):
    t = np.random.default_rng(sum(grid)).integers(0, 4, grid[0] * grid[1] * grid[2])
    return np.array([0.01, 0.05, 0.2, 0.1])[t], np.array([1.0, 2.0, 0.5, 1.3])[t]


def _forward(rte, grid, prec, mode, L=1, thresh=None):
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=thresh) as ctx:
        mua, mus = _medium(grid)

        def run():
            ctx.set_medium_voxel(mua, mus)
            ctx.forward(rte.Source(kind=rte.SRC_COLUMN), rte.Stop(rte.STOP_FIXED, 6), want_W=False)
        return _ms(run)


def _gradient(rte, grid, prec, mode):
    with rte.Context(*grid, dx=0.1, nL=1, g=0.8, precision=prec, kernel_mode=mode) as ctx:
        mua, mus = _medium(grid)
        srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_FIXED, 6), rte.Detector(nbins=2, faces=63)
        ctx.set_medium_voxel(mua * 1.05, mus)
        target = ctx.detector_flux(srcs, stop, det)
        ctx.set_medium_voxel(mua, mus)
        return _ms(lambda: ctx.gradient(srcs, stop, det, target))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,cube,factor", [((1, 1, 1000), 10, 40), ((2, 2, 700), 14, 40)])
def test_tall_columns(rte, grid, cube, factor, prec):
    """Recomputed, 1x1x1000 mixed: 1583 ms by one CTA, 6 ms with its blocks of z as units; 10^3 takes 1.2 ms."""
    a = _forward(rte, grid, prec, rte.KERNEL_RECOMPUTE)
    assert a < factor * _forward(rte, (cube,) * 3, prec, rte.KERNEL_RECOMPUTE)


@pytest.mark.parametrize("prec", [0, 1])
def test_gradient_of_a_tall_column(rte, prec):
    """1x1x600 with recomputed path integrals, mixed: 429 ms by one CTA, 16 ms now; 8^3 takes 2 ms."""
    a = _gradient(rte, (1, 1, 600), prec, rte.KERNEL_RECOMPUTE)
    assert a < 40 * _gradient(rte, (8, 8, 8), prec, rte.KERNEL_RECOMPUTE)


@pytest.mark.parametrize("prec", [0, 1])
def test_limited_coupling(rte, prec):
    """Recomputed path integrals at 33^3 with coupling over 2.5 voxels against coupling over the whole grid: 0.4 of the
    time while rows without coupled pairs were computed, 0.1 by a walk per coupled pair and less now."""
    n = (33, 33, 33)
    a = _forward(rte, n, prec, rte.KERNEL_RECOMPUTE, thresh=0.25)
    assert a < 0.25 * _forward(rte, n, prec, rte.KERNEL_RECOMPUTE)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [1, 2])
def test_flat_grid(rte, prec, mode):
    """110x110x1 against 23^3: 50 and 150 times its time with z columns (kernel stored, recomputed), 1 to 7 now."""
    a = _forward(rte, (110, 110, 1), prec, mode)
    assert a < 20 * _forward(rte, (23, 23, 23), prec, mode)
