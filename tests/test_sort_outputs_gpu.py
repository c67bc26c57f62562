"""rq_sort_rays into buffers at any byte: the outputs are the same wherever they
lie, on a float4 boundary or off it, and nothing beside them is written."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 257, 5003])
@pytest.mark.parametrize("ray_off, perm_off", [(0, 0), (16, 4), (4, 0), (8, 2), (1, 3), (17, 1)])
def test_sort_output_alignment(rq, n, ray_off, perm_off):
    import torch
    rng = np.random.default_rng(n)
    rays = torch.from_numpy(rng.uniform(-1, 1, (n, 8)).astype(np.float32)).cuda()
    lo, hi = (C.c_float * 3)(-1, -1, -1), (C.c_float * 3)(1, 1, 1)
    ctx = rq.Context()
    out, perm = torch.empty_like(rays), torch.empty(n, dtype=torch.int32, device="cuda")
    assert rq.lib.rq_sort_rays(ctx._h, rays.data_ptr(), n, lo, hi, out.data_ptr(), perm.data_ptr(), None) == 0
    b_out = torch.full((32 * n + 64,), 7, dtype=torch.uint8, device="cuda")
    b_perm = torch.full((4 * n + 64,), 7, dtype=torch.uint8, device="cuda")
    assert rq.lib.rq_sort_rays(ctx._h, rays.data_ptr(), n, lo, hi, b_out.data_ptr() + ray_off,
                               b_perm.data_ptr() + perm_off, None) == 0
    for got, off, want in ((b_out, ray_off, out), (b_perm, perm_off, perm)):
        got, want = got.cpu().numpy(), want.cpu().numpy().reshape(-1).view(np.uint8)
        assert np.array_equal(got[off:off + want.size], want)
        assert (got[:off] == 7).all() and (got[off + want.size:] == 7).all()
