"""The radiance cache's calls where they are cut or change loads: counts around
a chunk, around a wave of the gradient scatter, and records that start on a
float and not on a vector boundary.

A query's prediction does not depend on the call it is part of, so cut and
whole calls are equal bit for bit. Gradients are the same sums in another
order: at most some 500 terms per entry at the coarsest level, relative L2
below 1e-4 as test_gpu_nrc.py allows against the oracle. (The oracle is no
reference for 10^4 records and more, nor is the mean over smaller calls: a
rectifier at zero, or a BF16 rounding under another 1 / count, goes the other
way for one of them.)
"""
import numpy as np
import pytest

from test_gpu_nrc import queries, radiance_field

pytestmark = pytest.mark.gpu

QUERY_CHUNK = 1 << 20
TRAIN_CHUNK = 1 << 18
WAVE = 148 * 128


@pytest.fixture(scope="module")
def cache():
    from hdcodex_b200 import RadianceCache
    with RadianceCache(0, log2_table_size=14, base_resolution=16, finest_resolution=512, seed=5) as c:
        mlp, grid = c.parameters()
        grid[:] = np.random.default_rng(4).uniform(-0.5, 0.5, grid.size)
        c.set_parameters(mlp, grid)
        yield c


def records(n, seed, offset=0):
    """Device records that start `offset` floats into their allocation."""
    import torch
    q = queries(n, seed)
    buffer = torch.zeros(q.size + 4, dtype=torch.float32, device="cuda")
    buffer[offset:offset + q.size] = torch.from_numpy(q).cuda().ravel()
    return q, buffer[offset:]


@pytest.mark.parametrize("n", [QUERY_CHUNK - 1, QUERY_CHUNK, QUERY_CHUNK + 129])
def test_queries_across_chunks(cache, n):
    import torch
    _, dq = records(n, n % 91)
    whole = torch.full((n,), float("nan"), device="cuda")
    cache.query(dq.data_ptr(), n, whole.data_ptr())
    cut = torch.full((n,), float("nan"), device="cuda")
    at = 0
    for part in (1, 127, 512, 513, n - 1153):
        cache.query(dq.data_ptr() + at * 48, part, cut.data_ptr() + at * 4)
        at += part
    assert at == n and torch.isfinite(whole).all() and torch.equal(whole, cut)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_records_on_a_float_boundary(cache, offset):
    import torch
    n = 1000
    q, aligned = records(n, 8)
    _, shifted = records(n, 8, offset)
    targets = torch.from_numpy(np.concatenate([np.zeros(offset, np.float32), radiance_field(q)])).cuda()
    a, b = torch.zeros(n, device="cuda"), torch.zeros(n + 1, device="cuda")
    cache.query(aligned.data_ptr(), n, a.data_ptr())
    cache.query(shifted.data_ptr(), n, b.data_ptr() + 4)
    assert torch.equal(a, b[1:])
    plain = targets[offset:].clone()
    one = cache.gradients(aligned.data_ptr(), plain.data_ptr(), n)
    two = cache.gradients(shifted.data_ptr(), targets.data_ptr() + 4 * offset, n)
    for x, y in zip(one, two):
        assert np.linalg.norm(x - y) / np.linalg.norm(x) < 1e-4


@pytest.mark.parametrize("n", [1, 129, WAVE - 1, WAVE, WAVE + 1, TRAIN_CHUNK, TRAIN_CHUNK + 129])
def test_gradients_add_up_over_waves_and_chunks(cache, n):
    """Every record twice: the mean over 2 n records is the one over n, its
    output gradients scaled by a power of two (the same BF16 roundings), and
    waves and chunks end at other records."""
    import torch
    q, _ = records(n, 17)
    y = radiance_field(q)
    once = (torch.from_numpy(q).cuda(), torch.from_numpy(y).cuda())
    twice = tuple(torch.cat([x, x]) for x in once)
    a = cache.gradients(once[0].data_ptr(), once[1].data_ptr(), n)
    b = cache.gradients(twice[0].data_ptr(), twice[1].data_ptr(), 2 * n)
    for x, r in zip(a, b):
        assert np.linalg.norm(r) > 0.0
        assert np.linalg.norm(x - r) / np.linalg.norm(r) < 1e-4
