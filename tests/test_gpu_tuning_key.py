"""A tuning is served to scenes whose renders launch the same kernels only."""
import copy

import pytest

from hdcodex_b200 import PathTracer, workloads

pytestmark = pytest.mark.gpu


def test_scenes_with_other_kernels_are_tuned_by_themselves():
    w, h, spp = 40, 24, 2
    coat = workloads.closed_box(width=w, height=h)  # the whole closure; lanes seldom part
    coat.scene.materials[0].coat = 0.5
    glass, walks = copy.deepcopy(coat), copy.deepcopy(coat)
    glass.scene.materials[0].transmission = 0.5
    walks.scene.materials[0].subsurface = 0.5
    for wl in (coat, glass, walks):
        for fresh in (True, False):
            with PathTracer(0) as t:
                t.set_scene(wl.scene)
                assert (t.autotune(wl.camera, w, h, 3, spp)["candidates"] > 0) == fresh
