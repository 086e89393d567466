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


@pytest.mark.parametrize("fit", [0, 1, 2, 3], ids=["none", "mean", "and sums", "and batch"])
def test_image_buffers(box, expected, fit):
    large = 512 * 512
    sizes = [16, 24, 16, 24]  # bytes per pixel: mean, XYZ sums, batch, batch XYZ
    with PathTracer(0) as t:
        t.set_scene(box.scene)
        t.render(box.camera, W, H, 0, 8, 1)
        used, _ = device_memory_usage(0)
        freed = W * H * sum(sizes[:fit + 1])  # the small image's buffers go one by one
        set_device_memory_limit(0, used - freed + large * sum(sizes[:fit]) + 4096)
        try:
            with pytest.raises(RuntimeError, match="OUT_OF_MEMORY"):
                t.render(box.camera, 512, 512, 0, 8, 1)
        finally:
            set_device_memory_limit(0, 0)
        img = t.render(box.camera, W, H, 0, 8, 1)
        xyz, samples = t.read_xyz()
        assert np.array_equal(img, expected[0]) and samples == 1 and np.isfinite(xyz).all() and xyz.max() > 0


@pytest.mark.parametrize("fit", [0, 1], ids=["none", "ids"])
def test_aov_buffers(box, fit):
    with PathTracer(0) as t:
        t.set_scene(box.scene)
        t.set_aovs(3)
        t.render(box.camera, W, H, 0, 8, 1)
        aovs = t.read_aovs(W, H)
        t.set_aovs(0)
        t.render(box.camera, 256, 256, 0, 8, 1)  # image buffers and path state of the larger size
        t.set_aovs(3)
        used, _ = device_memory_usage(0)
        set_device_memory_limit(0, used - 4 * W * H * (fit + 1) + 4 * 256 * 256 * fit + 4096)
        try:
            with pytest.raises(RuntimeError, match="OUT_OF_MEMORY"):
                t.render(box.camera, 256, 256, 0, 8, 1)
        finally:
            set_device_memory_limit(0, 0)
        t.render(box.camera, W, H, 0, 8, 1)
        for got, want in zip(t.read_aovs(W, H), aovs):
            assert np.array_equal(got, want)
