"""AO rays and the AO reduction at the sizes where their blocks and lane
groups end: surfels that share a block or span several, every lane count of
the reduction, and ray buffers that are only 16-byte aligned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _surfels(n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.normal(size=(n, 4)).astype(np.float32)
    nrm = rng.normal(size=(n, 4)).astype(np.float32)
    nrm[:, :3] /= np.linalg.norm(nrm[:, :3], axis=1, keepdims=True)
    nrm[::7, :3] = 0.0  # no surface: an empty ray
    return pos, nrm, rng.uniform(0.1, 2.0, n).astype(np.float32)


@pytest.mark.parametrize("n,spp", [(1, 1), (255, 1), (256, 1), (257, 1), (1000, 3), (113, 37), (9, 255), (9, 256),
                                   (9, 257), (3, 1000)])
def test_aorays_block_edges(rq, po, n, spp):
    import torch
    pos, nrm, rad = _surfels(n, n + spp)
    dev = [torch.from_numpy(x).cuda() for x in (pos, nrm, rad)]
    buf = torch.full((n * spp * 8 + 8,), 3.0, device="cuda")
    out = buf[:n * spp * 8].view(-1, 8)
    rq.aorays(*dev, spp, 2 ** 40 + 11, 0.001, 3.0, 0.5, out=out)
    got = out.cpu().numpy()
    want = po.aorays(pos, nrm, rad, spp, 2 ** 40 + 11, 0.001, 3.0, 0.5)
    # float32 directions and origins from the same numbers: the tolerance of test_raygen_gpu.py
    assert np.abs(got - want).max() <= 2e-5 * max(1.0, np.abs(want[:, :3]).max())
    assert (buf[n * spp * 8:] == 3.0).all()
    # a buffer aligned to 16 bytes only: the same bytes
    half = torch.full((n * spp * 8 + 8,), 3.0, device="cuda")
    off = half[4:4 + n * spp * 8].view(-1, 8)
    assert off.data_ptr() % 32 == 16
    rq.aorays(*dev, spp, 2 ** 40 + 11, 0.001, 3.0, 0.5, out=off)
    assert torch.equal(off.view(torch.int32), out.view(torch.int32))
    assert (half[:4] == 3.0).all() and (half[4 + n * spp * 8:] == 3.0).all()


@pytest.mark.parametrize("spp", [1, 2, 7, 8, 15, 16, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 300])
@pytest.mark.parametrize("n", [1, 31, 1025])
def test_ao_reduce_lane_groups(rq, spp, n):
    import torch
    g = torch.Generator().manual_seed(spp * 7 + n)
    ids = torch.randint(-1, 3, (n * spp,), generator=g, dtype=torch.int32)
    hits = torch.zeros((n * spp, 4), dtype=torch.int32)
    hits[:, 1] = ids
    got = rq.ao_reduce(hits.view(torch.float32).cuda(), n, spp).cpu()
    want = (ids.view(n, spp) != -1).sum(1).float() / spp
    assert torch.equal(got, want)
