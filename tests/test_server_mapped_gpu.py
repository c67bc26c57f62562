"""Bake requests whose arrays the server reads and writes in place (pinned) and
those it copies (pageable, 4-byte aligned, many surfels, many rays per
surfel): the same AO bit for bit, in one burst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(x, shift=0):
    import torch
    n = x.size
    buf = torch.empty(n + shift, dtype=torch.float32, pin_memory=True)
    out = buf.numpy()[shift:].reshape(x.shape)
    out[...] = x
    return out


def test_mapped_and_copied_requests_agree(rq):
    import torch
    from cwbvh_b200 import workloads as W
    scenes = [W.upload(*W.scene_of_size(60 + k, 4000), rq.CWBVH) for k in range(2)]
    srv = rq.Server(hbm_budget_bytes=1 << 30, query=rq.ANY, streams=2, max_batch_rays=1 << 20)
    ids = [srv.add_scene(d.scene) for d in scenes]
    reqs, want = [], []
    ctx = rq.Context()
    for k, (n, spp) in enumerate([(1, 1), (1, 64), (7, 37), (255, 1), (257, 3), (1000, 32), (300, 256), (300, 257),
                                  (40, 1000), (32768, 2), (32769, 2), (40000, 4)]):
        ds = scenes[k % 2]
        dev = rq.sample_surfels(ds.vertices, ds.indices, n, 70 + k)
        seed, tmin, tmax = 2 ** 33 + k, 1e-4 * ds.diag, 0.1 * ds.diag
        rays = rq.aorays(*dev, spp, seed, tmin, tmax, 0.5)
        want.append(rq.trace_ao(ctx, ds.scene, rays, spp).cpu().numpy().astype(np.float32) / np.float32(spp))
        host = [x.cpu().numpy() for x in dev]
        for arrays in (host, [_pinned(x) for x in host], [_pinned(x, 1) for x in host],
                       [_pinned(host[0]), host[1], None]):
            for out in (np.full(n + 3, 9.0, np.float32), _pinned(np.full(n + 3, 9.0, np.float32))):
                t = srv.submit_bake(ids[k % 2], *arrays, spp, seed, tmin, tmax, 0.5, out)
                reqs.append((t, k, n, out, arrays))
    ctx.check()
    for t, k, n, out, _ in reqs:
        srv.wait(t)
        # the surfels' radius is 0, so a request without radii has the same rays
        assert np.array_equal(out[:n], want[k]), k
        assert (out[n:] == 9.0).all()
    srv.close()
