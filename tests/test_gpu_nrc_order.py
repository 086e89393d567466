"""The order in which training adds up the gradients of a hash-grid entry.

A block of the training kernel takes tiles of 128 records, one per
multiprocessor apart, and adds all of a tile's gradients before any of its next
tile's. The FP32 sum of an entry depends on that order, and Adam passes the
sum's rounding on to parameters whose gradient nearly cancels.

The network is set up so that the order shows in every bit: feature 0 of each
level reaches the output through ones, the records' direction gates it
(a record whose unit is off has no gradient at all), all records lie in the
grid's corner, and the table is zero, so that the prediction is 1 and the
gradient a multiple of 1 - target. Records of the last warp of the first
block's tiles have the gradient a, one record of the first warp of that block's
last tile has 2^27 a. In the tiles' order the sum of the small gradients is
exact (a has eight bits) and the large one is added to it, with one rounding; a
small gradient that comes after the large one is lost (a is below half a unit
in the last place of 2^27 a). The expected sum is therefore exact: no
tolerance.
"""
import numpy as np
import pytest

import nrc_oracle as N

pytestmark = pytest.mark.gpu

TILE = 128
LOG2 = 10
BIG = 2.0 ** 27


@pytest.mark.parametrize("tiles", [2, 13])
def test_a_tiles_gradients_are_added_before_the_next_tiles(tiles):
    import torch
    from hdcodex_b200 import RadianceCache
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = (sms * (tiles - 1) + 1) * TILE
    q = np.zeros((count, 12), np.float32)
    q[:, 3] = -1.0
    targets = np.zeros(count, np.float32)
    small = np.concatenate([np.arange(96, 128) + t * sms * TILE for t in range(tiles - 1)])
    large = (tiles - 1) * sms * TILE
    q[small, 3] = 1.0
    q[large, 3] = 1.0
    targets[large] = -BIG  # 1 - target rounds to 2^27
    mlp = np.zeros(N.LAYER_OFFSET[4] + N.LAYER_ROWS[4] * N.WIDTH, np.float32)
    mlp[[2 * level for level in range(16)]] = 1.0  # row 0 of the first layer: feature 0 of each level,
    mlp[32] = 1.0                                  # and the direction's x
    for layer in range(1, 5):
        mlp[N.LAYER_OFFSET[layer]] = 1.0
    with RadianceCache(0, log2_table_size=LOG2, base_resolution=16, finest_resolution=512, seed=1) as cache:
        cache.set_parameters(mlp, np.zeros(cache.grid_parameter_count, np.float32))
        dq, dt = torch.from_numpy(q).cuda(), torch.from_numpy(targets).cuda()
        # The gradient of a record with prediction 1 and target 0, in BF16.
        f = np.float32
        a = N.bf16(f(2.0) / (f(1.0) + f(0.01)) * (f(1.0) / f(count)))
        expected = f(f(a * f(len(small))) + f(a * f(BIG)))
        for _ in range(8):
            _, grid = cache.gradients(dq.data_ptr(), dt.data_ptr(), count)
            got = grid.reshape(16, 1 << LOG2, 2)[:, 0, 0]
            assert (got == expected).all(), (got, expected)
