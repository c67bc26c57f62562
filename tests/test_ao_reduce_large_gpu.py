"""ao_reduce at the most rays a surfel can have, where the step past the last
one leaves 31 bits (34 GB of hits; one warp adds them up in about eight seconds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_most_rays_per_surfel(rq):
    import torch
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 34 GB of device memory with room to spare")
    n = 2 ** 31 - 1
    hits = torch.full((n, 4), -1, dtype=torch.int32, device="cuda")
    hits[:1000, 1] = 5
    hits[n // 2:n // 2 + 2 ** 20, 1] = 0
    hits[-7:, 1] = 3
    ao = rq.ao_reduce(hits.view(torch.float32), 1, n).item()
    del hits
    torch.cuda.empty_cache()
    assert ao == float(np.float32(1007 + 2 ** 20) / np.float32(n))
