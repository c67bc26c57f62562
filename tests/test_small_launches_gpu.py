"""CWBVH launches small enough for several lanes to a ray (the default launch
of a few ten thousand rays or fewer): hits bit-identical to the oracle's, at
the edges of the kernel's blocks and of the ranges that choose 8, 4 or one
lane per ray."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(rq):
    import torch
    from cwbvh_b200 import workloads as W
    V, I = W.heightfield_boxes(5)
    ds = W.upload(V, I, rq.CWBVH)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rays = W.ao_rays(ds, 270 * sms, seed=31, tmax_scale=1.0).cpu().numpy()
    rays[::5, 3] = 0.0      # tmin = 0 and < 0 beside ordinary rays
    rays[1::7, 3] = -0.25
    return ds, rays, sms


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 4096, (128, 0), (128, 1), (270, 0)], ids=str)
def test_small_launch_bit_exact(rq, po, scene, n, query):
    import torch
    ds, rays, sms = scene
    n = n if isinstance(n, int) else n[0] * sms + n[1]
    r = np.ascontiguousarray(rays[:n])
    hits = torch.full((n + 8, 4), 5.0, device="cuda")
    ctx = rq.Context()
    rq.trace(ctx, ds.scene, torch.from_numpy(r).cuda(), hits, query, count=n)
    ctx.check()
    got = hits.cpu().numpy()
    want = po.trace(rq.CWBVH, ds.host.nodes, ds.host.woop, r, query == rq.ANY)
    assert np.array_equal(got[:n].view(np.uint32), want.view(np.uint32))
    assert (got[n:] == 5.0).all()


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("sizes", [(1, 0, 17, 300), (7000, 1, 12000, 5000)], ids=["lanes8", "lanes4"])
def test_small_batch_bit_exact(rq, po, sizes, query):
    import torch
    from cwbvh_b200 import workloads as W
    ctx = rq.Context()
    items, want = [], []
    for k, n in enumerate(sizes):
        V, I = W.scene_of_size(40 + k, (1, 50, 900, 20000)[k])
        ds = W.upload(V, I, rq.CWBVH)
        rays = W.ao_rays(ds, max(n, 1), seed=50 + k, tmax_scale=1.0)[:n].contiguous()
        items.append((ds.scene, rays, torch.full((n, 4), 5.0, device="cuda")))
        want.append(po.trace(rq.CWBVH, ds.host.nodes, ds.host.woop, rays.cpu().numpy(), query == rq.ANY) if n else None)
    for sort in (-1, 0):
        b = rq.Batch(ctx, items, query, sort_threshold=sort)
        b.run()
        ctx.check()
        for (_, _, h), w in zip(items, want):
            if w is not None:
                assert np.array_equal(h.cpu().numpy().view(np.uint32), w.view(np.uint32))
                h.fill_(5.0)
        b.close()


def test_small_ao_counts(rq, po, scene):
    import torch
    ds, rays, _ = scene
    r = np.ascontiguousarray(rays[:37 * 111])
    ctx = rq.Context()
    got = rq.trace_ao(ctx, ds.scene, torch.from_numpy(r).cuda(), 37).cpu().numpy()
    ctx.check()
    want = po.trace(rq.CWBVH, ds.host.nodes, ds.host.woop, r, True)
    assert np.array_equal(got, (want[:, 1].view(np.int32) >= 0).reshape(-1, 37).sum(1))
