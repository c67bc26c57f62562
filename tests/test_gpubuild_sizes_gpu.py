"""GPU builds at the sizes where their stages change hands: one block does the
last clustering rounds from 2,048 clusters on, tiles hold 256 clusters, a
node's children share eight lanes.  Every triangle is stored once, the kernels
equal the oracle on the tree bit for bit, and the answers are the host
build's."""
import numpy as np
import pytest

from adjudicate import _explained, prim_ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1], ids=["lbvh", "ploc"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 255, 2047, 2048, 2049, 2305, 4097, 20001])
def test_build_sizes(rq, po, n, method):
    import torch
    from cwbvh_b200 import workloads as W
    V, I = W.scene_of_size(n, n + n // 8 + 100)
    assert I.shape[0] >= n
    I = np.ascontiguousarray(np.random.default_rng(n).permutation(I)[:n])
    v, i = torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda()
    for passes in (0, 2):
        sc = rq.Scene.build_gpu(v, i, optimize_passes=passes, method=method)
        nodes, woop, prim = sc.download()
        assert np.array_equal(np.sort(prim.reshape(-1, 3)[:, 0]), np.arange(n))
        assert (prim.reshape(-1, 3)[:, 1:] == -1).all()
        hb = rq.HostBVH(V, I, rq.CWBVH)
        ds = W.DeviceScene(rq.CWBVH, hb, sc, v, i, W.diag(V), n)
        rays = W.ao_rays(ds, 3000, seed=n + 5, tmax_scale=1.0)
        ctx = rq.Context()
        hits = torch.empty((3000, 4), device="cuda")
        rq.trace_ordered(ctx, sc, rays, hits, rq.CLOSEST)
        ctx.check()
        r, got = rays.cpu().numpy(), hits.cpu().numpy()
        want = po.trace(rq.CWBVH, nodes, woop, r, False)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        host = po.trace(rq.CWBVH, hb.nodes, hb.woop, r, False)
        g, h = prim_ids(got, prim), prim_ids(host, hb.prim_index)
        bad = [k for k in np.nonzero(g != h)[0] if not _explained(po, r[k], V, I, (int(g[k]), int(h[k])))]
        assert not bad, bad[:5]
