"""Grids of few layers, solved with columns along x or y: the operator with exact directions in every order, precision and
kernel mode, complex mu_t, its adjoint, recorded series, batches, the gradient and the Fisher matrix; the table model's
pair-by-pair form.

Tolerances: FP64 1e-11 relative L2 against the FP64 oracle (sums of up to N terms of 1e-16 each, the orthogonal change of
coefficients adds a few 1e-16), mixed precision 1e-5, the method's bound; graph and batch against single solves the same
sums in another order; gradient and Fisher matrix against central differences of converged solves (step h = 1e-4: h^2
times the ratio of third to first derivatives, some tens at these optical depths)."""
import numpy as np
import pytest

from conftest import real_to_complex, rel

pytestmark = pytest.mark.gpu

GRIDS = [(64, 4, 1, 3), (4, 65, 1, 5), (129, 2, 2, 7), (3, 90, 6, 2), (30, 9, 9, 1), (1, 256, 1, 4), (300, 1, 1, 6), (20, 13, 3, 0), (64, 8, 12, 2)]
_REF = {}


def _medium(N, seed=3):
    t = np.random.default_rng(seed).integers(0, 4, N)
    return np.array([0.01, 0.05, 0.2, 0.1])[t], np.array([1.0, 2.0, 0.5, 1.3])[t]


def _params(oracle, ctx, grid, L, mode, kappa=0.0):
    d = [0.1] * 3
    if mode == oracle.MODE_FIM:  # the table model's extents are float fields, as the reference's
        f, g = np.float32, ctx.cfg
        d = [(float(f(b)) - float(f(a))) / n for a, b, n in zip((g.x_min, g.y_min, g.z_min), (g.x_max, g.y_max, g.z_max), grid)]
    return oracle.params(*grid, *d, L, 0.8, 1.0, ctx.cfg.prop_thresh, mode=mode, x_min=ctx.cfg.x_min,
                         y_min=ctx.cfg.y_min, z_min=ctx.cfg.z_min, **(dict(ssv=1, kappa=kappa) if mode == 0 else {}))


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("prec,tol", [(0, 1e-11), (1, 1e-5)])
@pytest.mark.parametrize("nx,ny,nz,L", GRIDS)
@pytest.mark.parametrize("mod", [0.0, 0.7])
def test_operator(rte, oracle, nx, ny, nz, L, prec, tol, mode, mod):
    grid, N, C = (nx, ny, nz), nx * ny * nz, (L + 1) ** 2
    mua, mus = _medium(N)
    rng = np.random.default_rng(N)
    W = real_to_complex(rng.standard_normal((N, C)), L)
    if mod:
        W = W + 1j * real_to_complex(rng.standard_normal((N, C)), L)
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode) as ctx:
        ctx.set_medium_voxel(mua, mus)
        ctx.set_modulation(mod)
        for flag in (1, 0):
            key = (grid, flag, mod)
            if key not in _REF:
                _REF[key] = oracle.apply(_params(oracle, ctx, grid, L, 0, mod), mua, mus, W, flag, 1)
            assert rel(ctx.prop_abs(W, flag, 1), _REF[key]) < tol


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("grid,L,model", [((64, 4, 1), 3, 0), ((3, 90, 2), 5, 0), ((64, 4, 2), 2, 1), ((4, 66, 1), 3, 1)])
def test_adjoint_is_the_transpose(rte, grid, L, model, prec, tol):
    N, C = grid[0] * grid[1] * grid[2], (L + 1) ** 2
    rng = np.random.default_rng(N)
    x, y = (rng.standard_normal((N, C)) + 1j * rng.standard_normal((N, C)) for _ in range(2))
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=rte.KERNEL_STORE, model=model) as ctx:
        ctx.set_medium_voxel(*_medium(N))
        a, b = np.vdot(y, ctx.prop_abs(x, 1, 0)), np.vdot(ctx.prop_abs_adjoint(y, 1), x)
    assert abs(a - b) < tol * np.linalg.norm(x) * np.linalg.norm(y)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("prec,tol", [(0, 1e-6), (1, 1e-5)])
@pytest.mark.parametrize("grid,L", [((44, 6, 1), 2), ((6, 44, 2), 3), ((128, 2, 1), 5), ((20, 14, 1), 7), ((16, 18, 3), 0)])
def test_table_model(rte, oracle, grid, L, prec, tol, mode):
    """Against the oracle, whose table mode walks the paths in FP32 as the reference does: 1e-6, as the table model's other
    operator test."""
    N, C = grid[0] * grid[1] * grid[2], (L + 1) ** 2
    mua, mus = _medium(N)
    W = real_to_complex(np.random.default_rng(N).standard_normal((N, C)), L)
    for thresh in (None, 0.25):
        with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, model=rte.MODEL_FIM,
                         prop_thresh=thresh) as ctx:
            ctx.set_medium_voxel(mua, mus)
            ref = oracle.apply(_params(oracle, ctx, grid, L, oracle.MODE_FIM), mua, mus, W, 1, 1)
            assert rel(ctx.prop_abs(W, 1, 1), ref) < tol


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 2e-6)])
@pytest.mark.parametrize("nx,ny,nz,L,model", [(44, 6, 1, 2, 1), (6, 88, 4, 3, 1), (20, 14, 1, 7, 1), (64, 4, 1, 5, 0),
                                              (4, 100, 2, 3, 0)])
def test_layers_of_a_thicker_grid(rte, nx, ny, nz, L, model, prec, tol):
    """A distribution that is zero but in nz layers, applied to a grid of ten (z columns): between those layers no path
    leaves them, so their rows are the flat grid's.  Voxels of 1/8 cm, exact in the table model's float extents."""
    N, C = nx * ny * nz, (L + 1) ** 2
    mua, mus = _medium(N)
    W = real_to_complex(np.random.default_rng(N).standard_normal((N, C)), L)
    k0 = 3 * nx * ny
    big = [np.full(nx * ny * 10, v) for v in (0.03, 0.9)]
    Wb = np.zeros((nx * ny * 10, C), complex)
    big[0][k0:k0 + N], big[1][k0:k0 + N], Wb[k0:k0 + N] = mua, mus, W
    out = []
    for grid, m, w in (((nx, ny, nz), (mua, mus), W), ((nx, ny, 10), big, Wb)):
        with rte.Context(*grid, dx=0.125, nL=L, g=0.8, precision=prec, kernel_mode=rte.KERNEL_STORE, model=model,
                         prop_thresh=50.0) as ctx:
            ctx.set_medium_voxel(*m)
            out.append(ctx.prop_abs(w, 1, 1))
    assert rel(out[0], out[1][k0:k0 + N]) < tol


@pytest.mark.parametrize("grid,L,model", [((30, 10, 2), 5, 0), ((5, 60, 1), 3, 0), ((44, 6, 1), 2, 1)])
@pytest.mark.parametrize("mode", [1, 2])
def test_batches_and_graphs(rte, grid, L, model, mode):
    mua, mus = _medium(grid[0] * grid[1] * grid[2])
    srcs = [rte.Source(pos_x=0.1 * x, kind=rte.SRC_COLUMN, mag=m) for x, m in ((0, 1), (-1, 2), (1, 0.5))]
    stop = rte.Stop(rte.STOP_FIXED, 5)
    with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=rte.PREC_MIXED, kernel_mode=mode, model=model) as ctx:
        ctx.set_medium_voxel(mua * 1.5, mus)
        ctx.forward_graph(srcs, 5)
        ctx.set_medium_voxel(mua, mus)
        tr, rf, _ = ctx.forward_graph(srcs, 5)
        b = ctx.forward_batch(srcs, stop)
        for q, s in enumerate(srcs):
            one = ctx.forward(s, stop)
            assert rel(b["W"][q], one["W"]) < 2e-6
            assert rel(b["trans"][q], one["trans"]) < 2e-6 and rel(tr[q], one["trans"]) < 2e-6 and rel(rf[q], one["ref"]) < 2e-6


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("grid,L,thresh", [((52, 5, 1), 3, None), ((4, 65, 2), 5, None), ((32, 9, 3), 1, 0.45)])
def test_gradient_and_fisher(rte, grid, L, thresh, mode):
    srcs, stop, det = [rte.Source()], rte.Stop(rte.STOP_REL_L2, 600, 1e-13), rte.Detector(nbins=2, faces=63)
    mua, mus = _medium(grid[0] * grid[1] * grid[2])
    rng = np.random.default_rng(5)
    da, ds, h = mua * rng.uniform(0, 1, mua.size), mus * rng.uniform(0, 1, mua.size), 1e-4
    out = []
    for prec in (rte.PREC_FP64, rte.PREC_MIXED):
        with rte.Context(*grid, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=mode, prop_thresh=thresh) as ctx:
            def flux(a, s):
                ctx.set_medium_voxel(a, s)
                return ctx.detector_flux(srcs, stop, det)
            if prec == rte.PREC_FP64:
                target = flux(mua * 1.05, mus * 0.97)
                f = [(flux(mua + s * h * da, mus), flux(mua, mus + s * h * ds)) for s in (1, -1)]
                num_a, num_s = ((f[0][q] - f[1][q]) / (2 * h) for q in (0, 1))
                loss = [[np.sum((x - target) ** 2) for x in y] for y in f]
            ctx.set_medium_voxel(mua, mus)
            _, ga, gs = ctx.gradient(srcs, stop, det, target)
            J = ctx.fisher(srcs, stop, det, np.stack([da, 0 * da]), np.stack([0 * ds, ds]), want_J=True)[1]
            out.append((ga, gs, J))
    ga, gs, J = out[0]
    for g, d, q in ((ga, da, 0), (gs, ds, 1)):
        assert abs(g @ d - (loss[0][q] - loss[1][q]) / (2 * h)) < 1e-5 * np.sum(np.abs(g * d))
    J = np.reshape(J, (-1, 2))
    assert rel(J[:, 0], np.ravel(num_a)) < 1e-6 and rel(J[:, 1], np.ravel(num_s)) < 1e-6
    assert all(rel(b, a) < 1e-5 for a, b in zip(*out))
