"""The last rays of a persistent CWBVH launch, which groups of four lanes take
over: bit-identical to the oracle where no triangles are postponed, adjudicated
where they are, at ray counts around the takeover (8 rays a warp) and with
stacks that have and have not spilled."""
import numpy as np
import pytest

from adjudicate import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(rq):
    from cwbvh_b200 import workloads as W
    V, I = W.heightfield_boxes(5)
    ds = W.upload(V, I, rq.CWBVH)
    rays = W.ao_rays(ds, 80000, seed=77, tmax_scale=1.0).cpu().numpy()
    return V, I, ds, rays


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("ratio", [-1.0, 0.2, 0.9])
@pytest.mark.parametrize("smem", [4, 8, 16])
def test_last_rays(rq, po, scene, smem, ratio, query):
    import torch
    V, I, ds, rays = scene
    ctx = rq.Context()
    for n in (1, 8, 9, 31, 33, 5000):
        r = np.ascontiguousarray(rays[n:2 * n])
        hits = torch.full((n + 8, 4), 5.0, device="cuda")
        rq.trace(ctx, ds.scene, torch.from_numpy(r).cuda(), hits, query, count=n,
                 launch=rq.Launch(64, 0, smem, ratio, 2, 8))
        ctx.check()
        got = hits.cpu().numpy()
        want = po.trace(rq.CWBVH, ds.host.nodes, ds.host.woop, r, query == rq.ANY)
        if ratio < 0:
            assert np.array_equal(got[:n].view(np.uint32), want.view(np.uint32))
        else:
            compare(po, r, got[:n], want, ds.host.prim_index, V, I, query == rq.ANY)
        assert (got[n:] == 5.0).all()


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
def test_last_rays_of_a_batch(rq, po, scene, query):
    """From 16 rays per thread on the any-hit batch takes its rays through the ring."""
    import torch
    V, I, ds, rays = scene
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    total = min(len(rays), 16 * 32 * sms + 777)
    cuts = [0, 1, 40000, 40000, total]
    ctx = rq.Context()
    items = [(ds.scene, torch.from_numpy(np.ascontiguousarray(rays[a:b])).cuda(),
              torch.full((b - a, 4), 5.0, device="cuda")) for a, b in zip(cuts, cuts[1:])]
    b = rq.Batch(ctx, items, query, launch=rq.Launch(32, 1, 4, -1.0, 0, 0))
    b.run()
    ctx.check()
    got = np.concatenate([h.cpu().numpy() for _, _, h in items])
    want = po.trace(rq.CWBVH, ds.host.nodes, ds.host.woop, np.ascontiguousarray(rays[:total]), query == rq.ANY)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    b.close()
