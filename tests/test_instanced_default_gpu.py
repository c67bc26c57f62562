"""The default instanced launch (no postponing) gives the oracle's hits bit for
bit, closest and any-hit, at counts that leave warps and blocks part filled."""
import numpy as np
import pytest

from instancing_common import make_instances, world_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def inst(rq):
    meshes, blas, M, bi, flat, tri_off = make_instances(rq, n_inst=700, seed=9)
    scenes = [rq.Scene.from_host(b) for b in blas]
    return blas, scenes, rq.Tlas(scenes, M, bi)


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("n", [1, 31, 129, 5000, 300_001])
def test_default_instanced_bit_exact(rq, po, inst, query, n):
    import torch
    blas, scenes, tlas = inst
    rays = world_rays(n, n + 3)
    hits = torch.full((n + 4, 4), 5.0, device="cuda")
    which = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    ctx = rq.Context()
    rq.trace_instanced(ctx, tlas, torch.from_numpy(rays).cuda(), hits, query, instance_out=which)
    ctx.check()
    want, wi = po.trace_instanced(tlas.buffers(), [(b.nodes, b.woop) for b in blas], rays, query == rq.ANY)
    assert np.array_equal(hits[:n].cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert np.array_equal(which.cpu().numpy(), wi)
    assert bool((hits[n:] == 5.0).all())
