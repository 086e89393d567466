"""Profiled renders take another route than ordinary ones: with stage times or
traversal counting the extension rays of a bounce and the shadow rays of the
one before are traced in launches of their own (with kernels of their own when
counting) instead of in one. Image and ray counts are the same, bit for bit."""
import numpy as np
import pytest

import ref_scenes as R
from hdcodex_b200 import PathTracer, workloads
from hdcodex_b200.tracer import PROFILE_COUNT_TRAVERSAL, PROFILE_STAGE_TIMES
from test_gpu_instancing import box_with_instances

pytestmark = pytest.mark.gpu


def scene_of(kind):
    if kind == "instanced":
        wl = box_with_instances(1, opacity=0.7)  # stochastic extension, threshold shadows
        return wl.scene, wl.camera
    if kind == "walks":
        wl = workloads.closed_box(40, 40)
        for m in wl.scene.materials:
            m.subsurface, m.subsurface_scale, m.subsurface_color = 1.0, 0.3, [0.9, 0.5, 0.3]
        return wl.scene, wl.camera
    scene = R.mesh_light_scene(1.0 if kind == "mesh light" else 0.0)
    scene.lights = R.analytic_lights()[:2] if kind == "lit" else []
    return scene, R.base_camera()


@pytest.mark.parametrize("bounces,wave", [(1, 0), (8, 0), (8, 3000)])
@pytest.mark.parametrize("kind", ["lit", "mesh light", "sun and sky", "instanced", "walks"])
def test_profiled_renders_are_the_same(kind, bounces, wave):
    scene, camera = scene_of(kind)
    w, h, spp = 45, 37, 3
    seen = {}
    with PathTracer(0) as t:
        t.set_scene(scene)
        t.set_wave_size(wave)
        for flags in (0, PROFILE_STAGE_TIMES, PROFILE_COUNT_TRAVERSAL, PROFILE_STAGE_TIMES | PROFILE_COUNT_TRAVERSAL):
            t.set_profiling(flags)
            seen[flags] = (t.render(camera, w, h, 0, bounces, spp), t.stats())
    image, stats = seen[0]
    assert stats["extension_rays"] > 0 and (kind == "walks" and bounces > 1) == (stats["subsurface_rays"] > 0)
    for flags, (img, st) in seen.items():
        assert np.array_equal(img, image), flags
        for key in ("extension_rays", "shadow_rays", "subsurface_rays"):
            assert st[key] == stats[key], (flags, key)
        assert (st["extension_node_visits"] > 0) == bool(flags & PROFILE_COUNT_TRAVERSAL)
