"""Device memory of GPU builds: scratch is kept for the next build while a scene
built on the device lives, and all of it goes back with the last such scene,
and after a build that was refused."""
import gc

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 50])
def test_memory_goes_back(rq, split):
    import torch
    from cwbvh_b200 import workloads as W
    V, I = W.scene_of_size(2, 400000)
    v, i = torch.from_numpy(V).cuda(), torch.from_numpy(I).cuda()
    bad = i.clone()
    bad[7, 2] = -1
    gc.collect()
    torch.cuda.synchronize()

    def free():
        return torch.cuda.mem_get_info()[0]

    def refused():
        with pytest.raises(rq.RQError):
            rq.Scene.build_gpu(v, bad, split_budget=split)

    rq.Scene.build_gpu(v, i, split_budget=split)  # loads the kernels
    refused()
    base = free()
    for _ in range(3):
        sc = rq.Scene.build_gpu(v, i, split_budget=split)
        assert free() < base
        del sc
        assert free() == base
        refused()
        assert free() == base
