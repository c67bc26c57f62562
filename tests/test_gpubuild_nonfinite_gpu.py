"""GPU builds of meshes whose boxes or box centres are not finite, so that the
octant rule has no cost to choose a child's slot by: every node and triangle
is still reached from the root exactly once, and triangles that can be hit are
hit where they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(case):
    from cwbvh_b200 import workloads as W
    V, I = W.scene_of_size(3, 4000)
    if case == "huge":      # finite, but lo + hi overflows
        V = V / np.abs(V).max() * np.float32(3e38)
    elif case == "nan":     # triangles without a finite vertex after the others
        bad = len(V) + np.arange(600).reshape(200, 3)
        V, I = np.concatenate([V, np.full((600, 3), np.nan)]), np.concatenate([I, bad])
    else:
        hit = np.random.default_rng(1).choice(len(V), 1 if case == "one_inf" else 40, replace=False)
        V[hit[::2], 0] = np.inf
        V[hit[1::2], 1] = -np.inf
    return np.ascontiguousarray(V, np.float32), np.ascontiguousarray(I, np.int32)


def _reached(nodes):
    """Nodes and triangle slots met on a walk from the root."""
    raw = nodes.view(np.uint8).reshape(-1, 80)
    level, seen, tris = np.array([0]), [], []
    while level.size:
        seen.append(level)
        b = raw[level]
        child = b[:, 16:20].copy().view(np.int32)[:, 0]
        first = b[:, 20:24].copy().view(np.int32)[:, 0]
        inner = ((b[:, 15:16] >> np.arange(8)) & 1).astype(bool)
        count = np.where(inner, 0, np.array([0, 1, 0, 2, 0, 0, 0, 3])[b[:, 24:32] >> 5])
        for k in range(3):
            r, s = np.nonzero(count > k)
            tris.append(first[r] + (b[r, 24 + s] & 31) + k)
        level = (child[:, None] + np.cumsum(inner, 1) - 1)[inner]
        assert ((level >= 0) & (level < len(raw))).all() and sum(x.size for x in seen) <= len(raw)
    return np.sort(np.concatenate(seen)), np.sort(np.concatenate(tris))


@pytest.mark.parametrize("method", [0, 1], ids=["lbvh", "ploc"])
@pytest.mark.parametrize("case", ["one_inf", "infs", "nan", "huge"])
def test_nonfinite_boxes(rq, case, method):
    import torch
    from cwbvh_b200 import workloads as W
    V, I = _mesh(case)
    v, i = torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda()
    for passes in (0, 2):
        sc = rq.Scene.build_gpu(v, i, optimize_passes=passes, method=method)
        nodes, _, prim = sc.download()
        seen, tris = _reached(nodes)
        assert np.array_equal(seen, np.arange(len(nodes) // 5))
        assert np.array_equal(tris, np.arange(len(I)))
        assert np.array_equal(np.sort(prim.reshape(-1, 3)[:, 0]), np.arange(len(I)))
        if case == "nan":
            n = len(I) - 200
            ds = W.upload(V[:-600], I[:n], rq.CWBVH)
            rays = W.ao_rays(ds, 5000, seed=8, tmax_scale=1.0)
            got, want = torch.empty((5000, 4), device="cuda"), torch.empty((5000, 4), device="cuda")
            ctx = rq.Context()
            rq.trace(ctx, sc, rays, got, rq.CLOSEST)
            rq.trace(ctx, ds.scene, rays, want, rq.CLOSEST)
            ctx.check()
            assert torch.equal(got[:, 0], want[:, 0])
