"""The column form of the pair operator and its kernel precompute at the sizes where they can go wrong: columns of
one voxel, columns padded to a whole group of destinations, columns longer than one run of sources or one block of
the precompute, a single row or column of voxels, limited coupling, every order, several slabs of the recompute
workspace.

Tolerances: FP64 1e-11 relative L2 against the FP64 oracle (sums of up to N terms of 1e-16 each, the angular
functions' trigonometric coefficients sum to 1.1 at most); mixed precision 1e-5, the method's bound."""
import numpy as np
import pytest

from conftest import real_to_complex, rel

pytestmark = pytest.mark.gpu

GRIDS = [(6, 5, 1, 3), (5, 3, 2, 5), (4, 5, 3, 4), (3, 2, 5, 7), (1, 6, 7, 2), (5, 1, 4, 6), (1, 1, 20, 1),
         (2, 1, 33, 5), (1, 2, 49, 3), (1, 1, 97, 5), (12, 11, 4, 0)]
_REF = {}


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("prec,tol", [(0, 1e-11), (1, 1e-5)])
@pytest.mark.parametrize("nx,ny,nz,L", GRIDS)
def test_column_operator(rte, oracle, nx, ny, nz, L, prec, tol, mode):
    rng = np.random.default_rng(nx * 1000 + ny * 100 + nz + L)
    N, C = nx * ny * nz, (L + 1) ** 2
    thresh = 0.07 * (nx + ny + nz) if L == 4 else None
    with rte.Context(nx, ny, nz, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=thresh) as ctx:
        p = oracle.params(nx, ny, nz, 0.1, 0.1, 0.1, L, 0.8, 1.0, ctx.cfg.prop_thresh, mode=rte.MODEL_EXACT, ssv=1,
                          x_min=ctx.cfg.x_min, y_min=ctx.cfg.y_min, z_min=ctx.cfg.z_min)
        tiss = rng.integers(0, 4, N)  # few distinct values: the oracle's self-voxel quadrature runs once for each
        mua, mus = np.array([0.01, 0.05, 0.2, 0.1])[tiss], np.array([1.0, 2.0, 0.5, 1.3])[tiss]
        ctx.set_medium_voxel(mua, mus)
        W = real_to_complex(rng.standard_normal((N, C)), L)
        key = (nx, ny, nz, L)
        if key not in _REF:
            _REF[key] = oracle.apply(p, mua, mus, W, 1, 1)
        assert rel(ctx.prop_abs(W, 1, 1), _REF[key]) < tol


@pytest.mark.parametrize("n,prec,tol", [(23, 0, 1e-12), (27, 1, 2e-6)])
def test_recompute_slabs_equal_the_stored_kernel(rte, n, prec, tol):
    """More pairs than the recompute workspace holds: the sources come in several slabs (the last one ragged)."""
    rng = np.random.default_rng(n)
    N, L = n ** 3, 1
    mua, mus = rng.uniform(0.005, 0.1, N), rng.uniform(0.5, 2.0, N)
    W = real_to_complex(rng.standard_normal((N, 4)), L)
    out = []
    for mode in (rte.KERNEL_STORE, rte.KERNEL_RECOMPUTE):
        with rte.Context(n, n, n, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode) as ctx:
            ctx.set_medium_voxel(mua, mus)
            out.append(ctx.prop_abs(W, 1, 0))
    assert rel(out[1], out[0]) < tol


@pytest.mark.parametrize("nx,nz,prec,tol", [(160, 64, 0, 1e-12), (200, 64, 1, 2e-6)])
def test_slabs_of_partial_rows_equal_the_stored_kernel(rte, nx, nz, prec, tol):
    """The workspace holds fewer columns than a row of the grid has, so slabs start and end within rows and some
    chunks of column pairs have no source in the slab."""
    rng = np.random.default_rng(nx)
    N, L = nx * 2 * nz, 1
    assert N * nz * (8, 4)[prec] * nx > 1 << 30  # one row of source columns is more than the workspace
    mua, mus = rng.uniform(0.005, 0.1, N), rng.uniform(0.5, 2.0, N)
    W = real_to_complex(rng.standard_normal((N, 4)), L)
    out = []
    for mode in (rte.KERNEL_STORE, rte.KERNEL_RECOMPUTE):
        with rte.Context(nx, 2, nz, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode) as ctx:
            ctx.set_medium_voxel(mua, mus)
            out.append(ctx.prop_abs(W, 1, 0))
    assert rel(out[1], out[0]) < tol


@pytest.mark.parametrize("nx,ny,nz,L", [(5, 4, 7, 1), (3, 2, 1, 2), (2, 1, 33, 3), (4, 3, 5, 4), (7, 6, 5, 5), (1, 2, 49, 5),
                                        (5, 3, 4, 6), (4, 4, 9, 7)])
@pytest.mark.parametrize("nsrc", [2, 3, 4])
def test_batched_right_hand_sides_equal_single_ones(rte, nx, ny, nz, L, nsrc):
    """Two right-hand sides of a thread against one; the difference is the order of FP32 sums."""
    rng = np.random.default_rng(nx * 100 + nz + L)
    N = nx * ny * nz
    mua, mus = rng.uniform(0.005, 0.1, N), rng.uniform(0.5, 2.0, N)
    srcs = [rte.Source(pos_x=0.1 * nx * x, kind=rte.SRC_COLUMN, mag=m) for x, m in ((0, 1), (-0.2, 2), (0.2, 0.5), (0.4, 3))][:nsrc]
    stop = rte.Stop(rte.STOP_FIXED, 4)
    with rte.Context(nx, ny, nz, dx=0.1, nL=L, g=0.8, precision=rte.PREC_MIXED, kernel_mode=rte.KERNEL_STORE) as ctx:
        ctx.set_medium_voxel(mua, mus)
        got = ctx.forward_batch(srcs, stop, want_W=True)["W"]
        for q, s in enumerate(srcs):
            want = ctx.forward(s, stop, want_W=True)["W"]
            assert rel(got[q], want) < 2e-6
