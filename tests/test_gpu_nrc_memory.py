"""A radiance cache whose device memory does not hold the query workspace is
created all the same and gives the same predictions."""
import numpy as np
import pytest

from hdcodex_b200 import RadianceCache
from hdcodex_b200.tracer import device_memory_usage, set_device_memory_limit
from test_gpu_nrc import queries, radiance_field

pytestmark = pytest.mark.gpu

WORKSPACE = (1 << 20) * 64  # bytes


@pytest.mark.parametrize("missing", [16, WORKSPACE])
def test_a_cache_without_the_query_workspace(missing):
    """`missing`: bytes that the budget lacks for the workspace, up to all of it."""
    import torch
    q = queries(1000, 6)
    dq, dy = torch.from_numpy(q).cuda(), torch.from_numpy(radiance_field(q)).cuda()
    outs = []
    before, _ = device_memory_usage(0)
    limit = 0
    try:
        for _ in range(2):
            set_device_memory_limit(0, limit)
            with RadianceCache(0, log2_table_size=12, finest_resolution=128, seed=9) as cache:
                whole = device_memory_usage(0)[0] - before
                out = torch.zeros(len(q), device="cuda")
                cache.query(dq.data_ptr(), len(q), out.data_ptr())
                outs.append(out.cpu().numpy())
                assert np.isfinite(cache.train(dq.data_ptr(), dy.data_ptr(), len(q), 1))
            if limit:
                assert whole == full - WORKSPACE
            full = whole
            limit = before + full - missing
    finally:
        set_device_memory_limit(0, 0)
    assert np.abs(outs[0]).max() > 0 and np.array_equal(outs[0], outs[1])
