"""Contexts on a device whose memory is nearly taken: automatic mode recomputes where the pair kernel does not fit, and goes
over to storing it when memory comes free."""
import contextlib

import pytest
import torch

from conftest import rel

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _left(nbytes):
    """About nbytes of device memory left."""
    torch.cuda.init()
    held = torch.empty(max(0, torch.cuda.mem_get_info()[0] - nbytes), dtype=torch.uint8, device="cuda")
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
