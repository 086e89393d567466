"""A render that runs out of device memory half way through its buffers leaves
nothing behind that a later render would take for whole buffers."""
import numpy as np
import pytest

from hdcodex_b200 import PathTracer, render_batch, workloads
from hdcodex_b200.tracer import device_memory_usage, set_device_memory_limit

pytestmark = pytest.mark.gpu

W, H = 64, 48
PATHS = W * H * 3


@pytest.fixture(scope="module")
def box():
    return workloads.closed_box(width=W, height=H)


@pytest.fixture(scope="module")
def expected(box):
    with PathTracer(0) as t:
        t.set_scene(box.scene)
        return [t.render(box.camera, W, H, 0, 8, spp) for spp in (1, 64)]


# Bytes of growth allowed per path of the larger render: none of its buffers
# (a path takes 352 bytes), and up to about half and nearly all of them.
@pytest.mark.parametrize("share", [4, 176, 340])
@pytest.mark.parametrize("then", ["small", "large", "batch"])
def test_path_state(box, expected, share, then):
    with PathTracer(0) as t:
        t.set_scene(box.scene)
        t.render(box.camera, W, H, 0, 8, 1)  # image buffers, and path state of one sample
        used, _ = device_memory_usage(0)
        set_device_memory_limit(0, used - PATHS * 340 + 64 * PATHS * share)
        try:
            with pytest.raises(RuntimeError, match="OUT_OF_MEMORY"):
                t.render(box.camera, W, H, 0, 8, 64)
        finally:
            set_device_memory_limit(0, 0)
        if then == "batch":
            img = np.zeros((H, W, 4), np.float32)
            render_batch([(t, box.camera, W, H, 0, 8, 64, img)])
        else:
            img = t.render(box.camera, W, H, 0, 8, 1 if then == "small" else 64)
        assert np.array_equal(img, expected[0 if then == "small" else 1])
