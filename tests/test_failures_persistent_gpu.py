"""The step limit and the stack limit of the persistent CWBVH kernel: in its own
loop (full warps) and in the takeover of a launch's last rays, which goes on
with the stacks it finds (at most 8 rays left in a warp), plain and in batches
with and without the ray ring.  A named launch shape keeps these launches from
the kernel with several lanes per ray, which the other failure tests reach."""
import numpy as np
import pytest

from test_failures_gpu import INNER0, INNER1, _valid_after, cw_node, rays_inside

pytestmark = pytest.mark.gpu

CYCLE = cw_node(0, 0, 0x01, {0: INNER0}, [0])                      # node 0 below itself: an endless walk
GROWING = np.concatenate([cw_node(0, 0, 0x03, {0: INNER0, 1: INNER1}, [0, 1])] * 2)  # and a stack that grows


def _rays(n, live):
    """`live` of 32 neighbouring rays start inside the node, the others pass by it."""
    r = rays_inside(n, seed=n + live)
    away = np.arange(n) % 32 >= live
    r[away, 0:3] = (-50.0, -50.0, -50.0)
    r[away, 4:7] = (-0.6, -0.8, 0.0)
    return r


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("n, live", [(5, 32), (64, 5), (64, 32), (100_000, 3), (100_000, 32)])
@pytest.mark.parametrize("block, smem, batch", [(64, 4, False), (64, 16, False), (256, 8, False), (32, 4, True)])
@pytest.mark.parametrize("case", ["steps", "stack"])
def test_limits_of_the_persistent_kernel(rq, case, block, smem, batch, n, live, query):
    import torch
    scene = rq.Scene.from_arrays(rq.CWBVH, CYCLE if case == "steps" else GROWING, np.zeros((3, 4), np.float32))
    # one block per SM in batches: 100,000 any-hit rays are enough for the ring
    launch = rq.Launch(block, 1 if batch else 0, smem, -1.0, 2, 8, 2000 if case == "steps" else 0)
    ctx = rq.Context()
    r = _rays(n, live)
    rays, hits = torch.from_numpy(r).cuda(), torch.full((n, 4), 5.0, device="cuda")
    if batch:
        rq.Batch(ctx, [(scene, rays, hits)], query, launch=launch).run()
    else:
        rq.trace(ctx, scene, rays, hits, query, launch=launch)
    with pytest.raises(rq.RQError, match="TIMEOUT" if case == "steps" else "STACK_OVERFLOW"):
        ctx.check()
    got = hits.cpu().numpy()
    assert (got[:, 1].view(np.int32) == -1).all() and np.array_equal(got[:, 0], r[:, 7])
    ctx.check()  # reported once
    _valid_after(rq, ctx)
