"""Several threads on one radiance cache: a query does not wait for another
thread's on another stream, and the kernel it takes then (which encodes its
records itself) gives the same bits as the ordinary pair of kernels."""
import threading
import time

import numpy as np
import pytest

from hdcodex_b200 import PathTracer, RadianceCache, workloads
from test_gpu_nrc import queries

pytestmark = pytest.mark.gpu

LONG = 1 << 27  # some 50 ms of queries


@pytest.fixture(scope="module")
def records():
    import torch
    yield torch.zeros(LONG * 12, device="cuda"), torch.zeros(LONG, device="cuda")
    torch.cuda.empty_cache()


def during_a_long_query(cache, records, call):
    """Runs call() while another thread's query is under way. Returns whether
    it came back before that query, and its result."""
    ended = []
    started = threading.Event()

    def long_query():
        started.set()
        cache.query(records[0].data_ptr(), LONG, records[1].data_ptr())
        ended.append(time.perf_counter())

    other = threading.Thread(target=long_query)
    other.start()
    started.wait()
    time.sleep(0.005)
    result = call()
    end = time.perf_counter()
    other.join()
    return end < ended[0], result


@pytest.mark.parametrize("n", [1, 127, 512, 513, 100_000])
def test_queries_beside_another_have_the_same_bits(records, n):
    import torch
    with RadianceCache(0, log2_table_size=14, finest_resolution=512, seed=5) as cache:
        mlp, grid = cache.parameters()
        grid[:] = np.random.default_rng(4).uniform(-0.5, 0.5, grid.size)
        cache.set_parameters(mlp, grid)
        q = torch.from_numpy(queries(n, 3)).cuda()
        alone, beside = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
        torch.cuda.synchronize()
        cache.query(q.data_ptr(), n, alone.data_ptr())
        during_a_long_query(cache, records, lambda: cache.query(q.data_ptr(), n, beside.data_ptr()))
        assert torch.isfinite(alone).all() and alone.abs().max() > 0 and torch.equal(alone, beside)


def test_a_render_with_the_cache_does_not_wait_for_another_threads_query(records):
    import torch
    wl = workloads.closed_box(16, 16)
    with PathTracer(0) as t, RadianceCache(0, log2_table_size=14, finest_resolution=256, seed=2) as cache:
        t.set_scene(wl.scene)
        t.set_radiance_cache(cache, prefix_bounces=2, training_paths=128, train_steps=1)
        t.render(wl.camera, 16, 16, 0, 3, 1)
        cache.query(records[0].data_ptr(), 1000, records[1].data_ptr())
        torch.cuda.synchronize()
        # A host that stalls one attempt does not decide.
        assert any(during_a_long_query(cache, records, lambda: t.render(wl.camera, 16, 16, 0, 3, 1))[0] for _ in range(5))
        t.set_radiance_cache(None)
