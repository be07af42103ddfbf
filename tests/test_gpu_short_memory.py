"""Contexts on a device whose memory is nearly taken: automatic mode recomputes where the pair kernel does not fit, and goes
over to storing it when memory comes free."""
import contextlib

import numpy as np
import pytest
import torch

from conftest import rel

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _left(nbytes):
    """About nbytes of device memory left."""
    torch.cuda.init()
    held, n = None, max(0, torch.cuda.mem_get_info()[0] - nbytes)
    while held is None:
        try:
            held = torch.empty(n, dtype=torch.uint8, device="cuda")
        except torch.cuda.OutOfMemoryError:  # the last pages may not be had in one piece
            n -= 4 << 20
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.mark.parametrize("prec", [0, 1])
def test_kernel_stored_after_a_graph_that_kept_none(rte, prec):
    """The graph is recorded while the kernel does not fit beside 1 GB; the eager solve after it finds room, and fills
    the kernel it allocates.  Tolerance as the graph tests."""
    n, T = 13, 5
    src, stop = rte.Source(kind=rte.SRC_COLUMN), rte.Stop(rte.STOP_FIXED, T)
    mua, mus, _ = rte.sphere_phantom(n, nspheres=2, seed=2, rmin=0.15, rmax=0.3)
    with rte.Context(n, n, n, dx=0.1, nL=2, g=0.8, precision=prec, kernel_mode=rte.KERNEL_AUTO) as ctx:
        with _left(900 << 20):
            ctx.set_medium_voxel(mua, mus)
            tr, rf, _ = ctx.forward_graph([src], T)
            few = ctx.device_bytes()
        got = ctx.forward(src, stop, want_W=False)
        assert ctx.device_bytes() - few >= (8, 4)[prec] * n ** 6  # the kernel is stored now
        assert rel(got["trans"], tr[0]) < 1e-9 and rel(got["ref"], rf[0]) < 1e-9
        ctx.set_medium_voxel(mua * 1.3, mus)
        a = ctx.forward_graph([src], T)
        b = ctx.forward(src, stop, want_W=False)
        assert rel(a[0][0], b["trans"]) < 1e-9 and rel(a[1][0], b["ref"]) < 1e-9


@pytest.mark.parametrize("n,prec,tol", [(23, 0, 1e-12), (27, 1, 2e-6)])
def test_workspace_cut_short(rte, n, prec, tol):
    """The workspace wants 1 GB and gets at most half of 700 MB: it stays where it is from solve to solve (the memory
    comes free after the first), a graph can be recorded on it, and a Fisher matrix of a mixed context shares it with
    its FP64 solves.  The sums of more slabs come in another order: tolerances as the slab tests of the operator."""
    T = 3
    src, stop, det = rte.Source(kind=rte.SRC_COLUMN), rte.Stop(rte.STOP_FIXED, T), rte.Detector(nbins=2, faces=63)
    mua, mus, _ = rte.sphere_phantom(n, nspheres=2, seed=2, rmin=0.15, rmax=0.3)
    out = []
    for short in (False, True):
        with rte.Context(n, n, n, dx=0.1, nL=1, g=0.8, precision=prec, kernel_mode=rte.KERNEL_RECOMPUTE) as ctx:
            with _left(700 << 20) if short else contextlib.nullcontext():
                ctx.set_medium_voxel(mua, mus)
                a = ctx.forward(src, stop)
                size = ctx.device_bytes()
            assert not short or size < 600 << 20
            g = [ctx.forward_graph([src], T) for _ in range(2)]
            assert ctx.device_bytes() == size
            F, J = ctx.fisher([src], stop, det, mua, 0 * mus, want_J=True)
            g.append(ctx.forward_graph([src], T))
            for tr, rf, _ in g:
                assert rel(tr[0], a["trans"]) < 1e-9 and rel(rf[0], a["ref"]) < 1e-9
            out.append((a["W"], J))
    assert rel(out[1][0], out[0][0]) < tol and rel(out[1][1], out[0][1]) < tol


@pytest.mark.parametrize("left", [2, 8, 20, 40, 70])
def test_context_after_a_failed_allocation(rte, left):
    """A batch, a gradient and a Fisher matrix that find no room fail with an error; the context keeps nothing of what it
    freed or half made: a single solve, and with room the refused calls, give what they gave before."""
    n, T = 21, 3
    srcs = [rte.Source(pos_x=0.2 * q, kind=rte.SRC_COLUMN) for q in (-1, 0, 1)]
    stop, det = rte.Stop(rte.STOP_FIXED, T), rte.Detector(nbins=2, faces=63)
    mua, mus, _ = rte.sphere_phantom(n, nspheres=2, seed=2, rmin=0.15, rmax=0.3)

    def calls(ctx):
        return (lambda: [ctx.forward_batch(srcs, stop)["W"]],
                lambda: list(ctx.gradient(srcs[:1], stop, det, np.zeros((1, 6, 2, 2)))[1:]),
                lambda: list(ctx.fisher(srcs[:1], stop, det, mua, 0 * mus, want_J=True)))

    with rte.Context(n, n, n, dx=0.1, nL=5, g=0.8, precision=rte.PREC_MIXED, kernel_mode=rte.KERNEL_STORE) as ctx:
        ctx.set_medium_voxel(mua, mus)
        want = [f() for f in calls(ctx)]
        one = ctx.forward(srcs[0], stop)["W"]
    with rte.Context(n, n, n, dx=0.1, nL=5, g=0.8, precision=rte.PREC_MIXED, kernel_mode=rte.KERNEL_STORE) as ctx:
        ctx.set_medium_voxel(mua, mus)
        ctx.forward(srcs[0], stop)
        refused = 0
        with _left(left << 20):
            for f in calls(ctx):
                try:
                    f()
                except rte.RteError:
                    refused += 1
                assert rel(ctx.forward(srcs[0], stop)["W"], one) < 2e-6
        assert refused > 0
        for f, w in zip(calls(ctx), want):
            for a, b in zip(f(), w):
                assert rel(a, b) < 1e-5
