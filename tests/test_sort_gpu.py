"""rq_sort_rays against a stable numpy sort of the same keys: block and tile
edges, buffers that are only 16-byte aligned, and outputs that overlap the
input."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LO, HI = (-1.0, -2.0, 0.0), (3.0, 2.0, 0.0)  # the z extent is empty


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    r = rng.normal(size=(n, 8)).astype(np.float32) * 2
    r[::13, 0] = np.inf
    r[1::17, 1] = np.nan
    r[2::5, 4] = -0.0
    return r


def _want(r):
    lo, hi = np.array(LO, np.float32), np.array(HI, np.float32)
    ext = hi - lo
    with np.errstate(all="ignore"):
        f = np.where(ext > 0, (r[:, :3] - lo) / np.where(ext > 0, ext, 1).astype(np.float32), 0).astype(np.float32)
    f = np.fmin(np.fmax(f, np.float32(0)), np.float32(1))
    q = np.minimum(511, (f * np.float32(512)).astype(np.uint32)).astype(np.uint64)
    m = np.zeros(len(r), np.uint64)
    for b in range(9):
        for a in range(3):
            m |= ((q[:, a] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - a)
    key = (m << np.uint64(3)) | ((r[:, 4] < 0) * 4 + (r[:, 5] < 0) * 2 + (r[:, 6] < 0)).astype(np.uint64)
    return np.argsort(key, kind="stable")


def _sort(rq, ctx, rays, n, out, perm):
    assert rq.lib.rq_sort_rays(ctx._h, rays, n, (C.c_float * 3)(*LO), (C.c_float * 3)(*HI), out, perm, None) == 0


@pytest.mark.parametrize("n", [1, 2, 255, 257, 1023, 1024, 1025, 4097, 100003])
def test_sort_matches_numpy(rq, n):
    import torch
    ctx = rq.Context()
    r = _rays(n, n)
    want = _want(r)
    for shift in (0, 4):  # floats: 32-byte and 16-byte aligned
        src = torch.zeros(8 * n + 8, device="cuda")
        src[shift:shift + 8 * n] = torch.from_numpy(r.reshape(-1))
        dst = torch.full((8 * n + 8,), 5.0, device="cuda")
        perm = torch.full((n + 1,), -9, dtype=torch.int32, device="cuda")
        _sort(rq, ctx, src[shift:].data_ptr(), n, dst[shift:].data_ptr(), perm.data_ptr())
        assert np.array_equal(perm[:n].cpu().numpy(), want) and int(perm[n]) == -9
        got = dst.cpu().numpy()
        assert np.array_equal(got[shift:shift + 8 * n].view(np.uint32), r[want].reshape(-1).view(np.uint32))
        assert (got[:shift] == 5.0).all() and (got[shift + 8 * n:] == 5.0).all()


def test_sort_in_place(rq):
    import torch
    n = 5003
    ctx = rq.Context()
    r = _rays(n, 3)
    want = _want(r)
    buf = torch.from_numpy(r).cuda()
    perm = torch.empty(n, dtype=torch.int32, device="cuda")
    _sort(rq, ctx, buf.data_ptr(), n, buf.data_ptr(), perm.data_ptr())
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(buf.cpu().numpy().view(np.uint32), r[want].view(np.uint32))
