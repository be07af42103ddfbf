"""Recorded series (rte_forward_graph) after the context's state has changed between two replays."""
import dataclasses

import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nsrc", [1, 4])
def test_replay_after_a_modulated_solve(rte, prec, nsrc):
    """A modulated solve tabulates angle rows of another layout in the same buffer; every replay of the graph recorded
    without modulation equals the eager solve.  Tolerance as the graph tests: the same kernels on the same inputs."""
    n, L, T = 9, 3, 6
    srcs = [rte.Source(pos_x=x, pos_y=y, kind=rte.SRC_COLUMN) for x, y in ((0, 0), (0.2, 0), (0, -0.2), (-0.1, 0.3))][:nsrc]
    mua, mus, _ = rte.sphere_phantom(n, nspheres=2, seed=1, rmin=0.15, rmax=0.3)
    with rte.Context(n, n, n, dx=0.1, nL=L, g=0.8, precision=prec, kernel_mode=rte.KERNEL_STORE) as ctx:
        ctx.set_medium_voxel(mua, mus)
        ref = ctx.forward_batch(srcs, rte.Stop(rte.STOP_FIXED, T), want_W=False)
        for k in range(4):
            tr, rf, _ = ctx.forward_graph(srcs, T)
            for b in range(nsrc):
                assert rel(tr[b], ref["trans"][b]) < 1e-9 and rel(rf[b], ref["ref"][b]) < 1e-9, (k, b)
            ctx.forward(dataclasses.replace(srcs[0], modulation=0.7), rte.Stop(rte.STOP_FIXED, T), want_W=False)
            ctx.set_modulation(0.0)
