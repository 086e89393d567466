"""Adam on parameters without gradient and moments: left alone where the
formula leaves them, and given what it gives where it does not (a decay of one
or a rate that is not finite: 0 / 0 and infinity times zero)."""
import numpy as np
import pytest

from hdcodex_b200 import RadianceCache
from test_gpu_nrc import queries, radiance_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,stays", [
    ({}, True), ({"epsilon": 0.0}, False), ({"beta1": 1.0}, False), ({"beta2": 1.0}, False), ({"learning_rate": float("inf")}, False),
], ids=["default", "epsilon 0", "beta1 1", "beta2 1", "rate infinite"])
def test_parameters_without_gradient(config, stays):
    import torch
    q = queries(256, 2)
    q[:, :3] = 0.25  # every record in one place: most of the table has no gradient
    dq, dy = torch.from_numpy(q).cuda(), torch.from_numpy(radiance_field(q)).cuda()
    with RadianceCache(0, log2_table_size=12, finest_resolution=128, seed=4, **config) as cache:
        mlp, before = cache.parameters()
        _, gradient = cache.gradients(dq.data_ptr(), dy.data_ptr(), len(q))
        cache.train(dq.data_ptr(), dy.data_ptr(), len(q), 1)
        _, after = cache.parameters()
    idle = gradient == 0.0
    assert idle.mean() > 0.9 and not idle.all()
    if stays:
        assert np.array_equal(after[idle], before[idle]) and (after[~idle] != before[~idle]).any()
    else:
        assert np.isnan(after[idle]).all()
