"""Bake requests with a radius of its own for every surfel, and requests cut into
pieces, through both input paths: arrays read in place (pinned) and arrays
copied (pageable, or too many surfels).  The AO equals that of the rays made,
traced and reduced at once, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(x):
    import torch
    return torch.empty(x.shape, dtype=torch.float32, pin_memory=True).copy_(torch.from_numpy(x)).numpy()


# surfels, rays each, rays per launch: whole requests around the most surfels that are read in place (several of them
# pass what a launch reads in place), and pieces of 4,000, 1 and 300 surfels with a last one of another size
@pytest.mark.parametrize("n, spp, cap", [(3, 7, 1 << 20), (8191, 2, 1 << 20), (8192, 2, 1 << 20), (8193, 2, 1 << 20),
                                         (32768, 2, 1 << 20), (32769, 2, 1 << 20), (9001, 16, 64000), (5, 33, 33),
                                         (1000, 256, 76800), (70001, 2, 40000)])
def test_radii_and_pieces(rq, n, spp, cap):
    import torch
    from cwbvh_b200 import workloads as W
    ds = W.upload(*W.scene_of_size(61, 4000), rq.CWBVH)
    pos, nrm, _ = (x.cpu().numpy() for x in rq.sample_surfels(ds.vertices, ds.indices, n, 5))
    # origins up to a tenth of the scene above the surface: another radius is another AO
    rad = np.random.default_rng(n).uniform(0.0, 0.1 * ds.diag, n).astype(np.float32)
    seed, tmin, tmax = 2 ** 34 + n, 1e-4 * ds.diag, 0.1 * ds.diag
    ctx = rq.Context()

    def reference(radius):
        r = None if radius is None else torch.from_numpy(radius).cuda()
        rays = rq.aorays(torch.from_numpy(pos).cuda(), torch.from_numpy(nrm).cuda(), r, spp, seed, tmin, tmax, 1.0)
        return rq.trace_ao(ctx, ds.scene, rays, spp).cpu().numpy().astype(np.float32) / np.float32(spp)

    want, want_none = reference(rad), reference(None)
    ctx.check()
    assert n < 100 or not np.array_equal(want, want_none)
    srv = rq.Server(hbm_budget_bytes=1 << 28, query=rq.ANY, streams=2, max_batch_rays=cap)
    sid = srv.add_scene(ds.scene)
    reqs = []
    p = [_pinned(x) for x in (pos, nrm, rad)]
    for arrays, w in ((p, want), ([pos, nrm, rad], want), ([p[0], p[1], rad], want), ([p[0], p[1], None], want_none)):
        for out in (_pinned(np.full(n + 3, 9.0, np.float32)), np.full(n + 3, 9.0, np.float32)):
            reqs.append((srv.submit_bake(sid, *arrays, spp, seed, tmin, tmax, 1.0, out), out, w))
    for t, out, w in reqs:
        srv.wait(t)
        assert np.array_equal(out[:n], w) and (out[n:] == 9.0).all()
    if n * spp > cap:
        assert srv.memory()["pieces"] >= len(reqs) * -(-n * spp // cap)
    srv.close()
