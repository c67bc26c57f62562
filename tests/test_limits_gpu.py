"""Node and triangle addresses at the very end of their buffers are read, the
next ones are errors: the trace kernels' limits at buffers of the smallest
sizes, for one and several lanes to a ray, plain and batched."""
import numpy as np
import pytest

from test_failures_gpu import LEAF1, cw_node, rays_inside

pytestmark = pytest.mark.gpu

WALL = np.array([[0, 0, 1, 1e30], [0, 0, 0, 0], [0, 0, 0, 0]], np.float32)  # a row triple nothing hits
END = np.array([[0x80000000, 0, 0, 0]], np.uint32).view(np.float32)         # a BVH2 leaf's terminator


def _status(rq, kind, nodes, woop, query, n, batch):
    import torch
    ctx = rq.Context()
    sc = rq.Scene.from_arrays(kind, nodes, woop)
    rays = torch.from_numpy(rays_inside(n)).cuda()
    hits = torch.full((n, 4), float("nan"), device="cuda")
    if batch:
        rq.Batch(ctx, [(sc, rays, hits)], query).run()
    else:
        rq.trace(ctx, sc, rays, hits, query)
    st = ctx.status()
    assert (hits[:, 1].view(torch.int32) == -1).all()
    return rq._native.STATUS.get(st, str(st))


@pytest.mark.parametrize("batch", [False, True], ids=["plain", "batch"])
@pytest.mark.parametrize("n", [64, 30_000, 100_000])
@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
def test_cwbvh_rows_at_the_end(rq, query, n, batch):
    # one leaf child whose triangle is number `tri_base`, in buffers of `rows` float4
    for rows, tri_base, ok in ((3, 0, True), (6, 1, True), (5, 1, False), (2, 0, False), (6, 2, False)):
        woop = np.tile(WALL, (3, 1))[:rows]
        node = cw_node(0, tri_base, 0, {0: LEAF1}, [0])
        got = _status(rq, rq.CWBVH, node, np.ascontiguousarray(woop), query, n, batch)
        assert ("BAD_SCENE" in got) != ok, (rows, tri_base, got)


@pytest.mark.parametrize("batch", [False, True], ids=["plain", "batch"])
@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
def test_bvh2_leaf_at_the_end(rq, query, batch):
    box = [-1e3, 1e3, -1e3, 1e3]

    def node(leaf):
        n = np.array([box, box, [-1e3, 1e3, -1e3, 1e3], [0, 0, 0, 0]], np.float32)
        n.view(np.int32)[3, :2] = [~leaf, ~leaf]
        return n
    for woop, leaf, ok in ((END, 0, True), (np.concatenate([WALL, END]), 0, True), (np.concatenate([WALL, END]), 3, True),
                           (END, 1, False), (WALL, 0, False), (WALL[:2], 0, False), (np.concatenate([END, END]), 1, True)):
        got = _status(rq, rq.BVH2, node(leaf), np.ascontiguousarray(woop), query, 5000, batch)
        assert ("BAD_SCENE" in got) != ok, (woop.shape, leaf, got)
