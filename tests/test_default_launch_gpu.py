"""The launch that rq_default_launch names and the unset one are the same kernel
launch, and the tuners can return it: compared by what a stream capture
records of each call."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


class KernelParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 6), ("smem", C.c_uint), ("params", C.c_void_p),
                ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _recorded(call):
    """(type, kernel, grid and block, shared memory) of each node of `call(stream)`."""
    import torch
    cu = C.CDLL("libcuda.so.1")

    def ok(status):
        assert status == 0, status
    s = torch.cuda.Stream()
    call(s)  # occupancy and kernel loading happen outside the capture
    torch.cuda.synchronize()
    graph, n = C.c_void_p(), C.c_size_t()
    ok(cu.cuStreamBeginCapture_v2(C.c_void_p(s.cuda_stream), 2))
    try:
        call(s)
    finally:
        end = cu.cuStreamEndCapture(C.c_void_p(s.cuda_stream), C.byref(graph))
    ok(end)
    ok(cu.cuGraphGetNodes(graph, None, C.byref(n)))
    nodes = (C.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, C.byref(n)))
    out = []
    for node in nodes:
        t = C.c_int()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(t)))
        p = KernelParams()
        if t.value == 0:
            ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)))
        out.append((t.value, p.func or 0, p.kern or 0, tuple(p.dims), p.smem))
    ok(cu.cuGraphDestroy(graph))
    return sorted(out)


@pytest.fixture(scope="module")
def scene():
    import cwbvh_b200 as rq
    from cwbvh_b200 import workloads as W
    ds = W.upload(*W.heightfield_boxes(5), rq.CWBVH)
    return ds, W.ao_rays(ds, 3 << 20, seed=3)


@pytest.mark.parametrize("query", [0, 1], ids=["closest", "any"])
@pytest.mark.parametrize("n", [64, 4096, 30_000, 100_000, 3 << 20])
def test_default_launch_is_the_unset_launch(rq, scene, n, query):
    import torch
    ds, rays = scene
    ctx = rq.Context()
    r, hits = rays[:n], torch.empty((n, 4), device="cuda")
    d = rq.default_launch(rq.CWBVH, query)
    other = rq.default_launch(rq.CWBVH, query)
    other.smem_stack = 16

    def plain(launch):
        return _recorded(lambda s: rq.trace(ctx, ds.scene, r, hits, query, launch=launch, stream=s))

    def batch(launch):
        b = rq.Batch(ctx, [(ds.scene, r, hits)], query, launch=launch)
        return _recorded(lambda s: b.run(s))

    for call in (plain, batch):
        unset = call(None)
        assert call(d) == unset and call(rq.Launch()) == unset
        assert call(other) != unset
    ctx.check()


def test_tuners_return_the_unset_launch_for_small_counts(rq, scene, tmp_path):
    """At 4,096 rays the kernel with several lanes per ray takes half the time
    of every named shape."""
    import torch
    ds, rays = scene
    ctx = rq.Context()
    cache = str(tmp_path / "tune")
    r, hits = rays[:4096].contiguous(), torch.empty((4096, 4), device="cuda")
    fields = ("block_size", "blocks_per_sm", "smem_stack", "postpone_ratio", "fetch_nd", "fetch_nw")

    def values(l):
        return [getattr(l, f) for f in fields]

    for query in (rq.CLOSEST, rq.ANY):
        want = values(rq.default_launch(rq.CWBVH, query))
        assert values(rq.autotune(ctx, ds.scene, r, hits, query, cache_path=cache)) == want
        assert values(rq.autotune(ctx, ds.scene, r, hits, query, cache_path=cache)) == want  # as cached
        items = [(ds.scene, r[:2048], hits[:2048]), (ds.scene, r[2048:], hits[2048:])]
        bp = rq.autotune_batch(ctx, items, query, cache_path=cache, stream=torch.cuda.Stream())
        assert values(bp.launch) == want
    # a choice cached without the kernels' revision, or with another, is not used
    lines = open(cache).read().splitlines()
    assert len(lines) == 4
    old = tmp_path / "old"
    for cut in (lambda k: k.replace("|r2", ""), lambda k: k.replace("|r2", "|r1")):
        old.write_text("\n".join(" ".join([cut(x.split()[0]), "64", *x.split()[2:]]) for x in lines) + "\n")
        l = rq.autotune(ctx, ds.scene, r, hits, rq.CLOSEST, cache_path=str(old))
        assert values(l) == values(rq.default_launch(rq.CWBVH, rq.CLOSEST))
