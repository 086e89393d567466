"""A render leaves its caller's path buffers as they are, so that a batch whose
graph could not be captured renders the same calls again on streams."""
import os
import subprocess

import numpy as np
import pytest

from hdcodex_b200 import PathTracer, render_batch, workloads

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_render_takes_its_path_buffers_unchangeable(tmp_path):
    """renderFrame accepts constant path buffers: compiled, not run."""
    from hdcodex_b200 import build as B
    src = tmp_path / "constant_buffers.cpp"
    src.write_text('#include "integrator.h"\n'
                   'void again(const hdcx::DeviceScene& s, const hdcx::FrameConst& f, const hdcx::PathBuffers& p,\n'
                   '           hdcx::FrameBuffers& fb) { hdcx::renderFrame(s, f, p, fb, nullptr, nullptr, false, nullptr); }\n')
    res = subprocess.run(["g++", "-std=c++20", "-fsyntax-only", "-I", B.INCLUDE, "-I", os.path.join(ROOT, "hdcodex_b200", "csrc"),
                          "-I", B.cuda_include(), str(src)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("bounces", [1, 8, 12])
def test_a_batch_that_cannot_be_captured_renders_on_streams(bounces):
    """The first batch with AOVs allocates them while it is captured, which
    ends the capture; the second one is captured."""
    from hdcodex_b200.tracer import batch_graph_stats
    spec = [(workloads.closed_box(width=w, height=h, spp=spp), w, h, spp) for w, h, spp in [(64, 48, 2), (96, 64, 3)]]
    expected = []
    for wl, w, h, spp in spec:
        with PathTracer(0) as t:
            t.set_scene(wl.scene)
            t.set_aovs(3)
            first = t.render(wl.camera, w, h, 0, bounces, spp)
            rays = t.stats()["extension_rays"], t.stats()["shadow_rays"]
            expected.append((first, rays, t.read_aovs(w, h), t.render(wl.camera, w, h, spp, bounces, 1)))
    tracers = [PathTracer(0) for _ in spec]
    try:
        for t, (wl, *_rest) in zip(tracers, spec):
            t.set_scene(wl.scene)
            t.set_aovs(3)
        images = [np.zeros((h, w, 4), np.float32) for _, w, h, _ in spec]
        before = batch_graph_stats(0)
        render_batch([(t, wl.camera, w, h, 0, bounces, spp, img) for t, (wl, w, h, spp), img in zip(tracers, spec, images)], 0, graph=True)
        assert batch_graph_stats(0) == before
        for t, img, (first, rays, aovs, _), (_, w, h, _) in zip(tracers, images, expected, spec):
            assert np.array_equal(img, first)
            assert (t.stats()["extension_rays"], t.stats()["shadow_rays"]) == rays
            for got, want in zip(t.read_aovs(w, h), aovs):
                assert np.array_equal(got, want)
        render_batch([(t, wl.camera, w, h, spp, bounces, 1, img) for t, (wl, w, h, spp), img in zip(tracers, spec, images)], 0, graph=True)
        assert sum(batch_graph_stats(0)) == sum(before) + 1
        for img, (*_, second) in zip(images, expected):
            assert np.array_equal(img, second)
    finally:
        for t in tracers:
            t.close()
