"""Path groups (the lanes of a sample that share a path travel as one queue
entry), the order in which waves take the image, and the kernels that depend
on both, at the sizes and settings where they change route.

The oracle traces every lane by itself in image order, so it is the general
form of each. Tolerance as in test_gpu_parity.py: at least 99% of pixels
bit-identical and an image-level relative L1 difference of at most 1e-3;
renders that differ only in how waves are cut must be equal bit for bit.
"""
import numpy as np
import pytest

import ref_scenes as R
from hdcodex_b200 import PathTracer, workloads
from hdcodex_b200.scene import SPHERE, Light

pytestmark = pytest.mark.gpu

MIN_IDENTICAL = 0.99
MAX_REL_L1 = 1e-3


@pytest.fixture(scope="module")
def gpu():
    t = PathTracer(0)
    yield t
    t.close()


def check(img, ref, what):
    same = float(np.all((img == ref) | (np.isnan(img) & np.isnan(ref)), axis=-1).mean())
    finite = np.isfinite(ref).all(axis=-1)
    denom = float(np.abs(ref[finite][..., :3]).sum()) + 1e-12
    rel = float(np.abs(img[finite][..., :3] - ref[finite][..., :3]).sum()) / denom
    assert same >= MIN_IDENTICAL and rel <= MAX_REL_L1, f"{what}: identical={same:.4f} relL1={rel:.2e}"


def both(oracle_lib, gpu, scene, w, h, spp, bounces=8, camera=None):
    o = oracle_lib.OracleTracer()
    o.set_scene(scene)
    camera = camera or R.base_camera()
    ref = o.render(camera, w, h, 0, bounces, spp)
    gpu.set_scene(scene)
    return gpu.render(camera, w, h, 0, bounces, spp), ref


# Blocks of 8 x 4 pixels, ragged at both edges; one pixel, one row, one column;
# more samples than a block of the accumulation has threads.
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (1, 13, 2), (13, 1, 3), (8, 4, 1), (9, 5, 2), (7, 3, 5), (33, 18, 3), (64, 31, 1), (3, 2, 300)])
def test_image_order_and_sample_counts(oracle_lib, gpu, w, h, spp):
    img, ref = both(oracle_lib, gpu, R.base_scene(), w, h, spp)
    check(img, ref, f"{w}x{h} {spp} spp")


@pytest.mark.parametrize("paths", [96, 3 * 33 * 17, 3 * 33 * 17 * 2, 5000])
def test_wave_cuts_give_the_same_image(gpu, paths):
    """Waves of part of a sample, one sample, two samples and a size that cuts rows."""
    with PathTracer(0) as small:
        small.set_scene(R.base_scene())
        whole = small.render(R.base_camera(), 33, 17, 0, 8, 4)
        small.set_wave_size(paths)
        cut = small.render(R.base_camera(), 33, 17, 0, 8, 4)
    assert np.array_equal(whole, cut)


def shadowed(color, distance, falloff, gamma):
    s = R.mesh_light_scene(0.0)  # a blocker in front of a receiver
    s.lights = [Light(id="/sphere", type=SPHERE, intensity=20.0, position=[1.6, 1.2, 0.5], radius=0.2, area=0.5026548,
                      shadow_color=color, shadow_distance=distance, shadow_falloff=falloff, shadow_falloff_gamma=gamma)]
    return s


@pytest.mark.parametrize("scene", [
    shadowed([0.0, 0.0, 0.0], -1.0, -1.0, 1.0),  # a blocked sample is zero
    shadowed([0.4, 0.1, 0.0], -1.0, -1.0, 1.0),  # it keeps the shadow's colour
    shadowed([0.0, 0.0, 0.0], 4.0, 2.0, 2.0),    # it falls off with the blocker's distance
    shadowed([0.2, 0.0, 0.3], 4.0, 2.0, 0.0),
], ids=["plain", "colour", "falloff", "colour-falloff"])
def test_blocked_light_samples(oracle_lib, gpu, scene):
    img, ref = both(oracle_lib, gpu, scene, 40, 40, 4)
    check(img, ref, "blocked light samples")


# Light-sample slots: one (lights), two (emissive triangles, with and without
# lights), three (neither: the fallback sun and sky).
@pytest.mark.parametrize("mesh,lights", [(False, True), (True, True), (True, False), (False, False)])
@pytest.mark.parametrize("full", [False, True])
def test_light_sample_slots(oracle_lib, gpu, mesh, lights, full):
    s = R.mesh_light_scene(1.0 if mesh else 0.0)
    s.lights = R.analytic_lights()[:2] if lights else []
    if full:
        s.materials[0].coat = 0.6
        s.materials[0].diffuse_model = 1
        s.materials[0].diffuse_roughness = 0.5
    img, ref = both(oracle_lib, gpu, s, 37, 29, 4)
    check(img, ref, f"mesh {mesh} lights {lights} full {full}")


@pytest.mark.parametrize("count", [1, 16, 17])
def test_lights_around_the_staged_number(oracle_lib, gpu, count):
    s = R.mesh_light_scene(0.0)
    s.lights = [Light(id=f"/l{i}", type=SPHERE, intensity=4.0 + i, position=[-1.5 + 0.2 * i, 1.5, -0.5 - 0.05 * i], radius=0.1,
                      area=0.1256637, color=[1.0, 0.3 + 0.04 * i, 0.2]) for i in range(count)]
    img, ref = both(oracle_lib, gpu, s, 33, 33, 4)
    check(img, ref, f"{count} lights")


def test_a_colour_that_is_not_finite_takes_the_general_kernel(oracle_lib, gpu):
    """Zero times an infinite colour is not zero: weights of zero do not
    select the kernel that leaves their lobes out."""
    s = R.mesh_light_scene(0.0)
    s.lights = R.analytic_lights()[1:2]
    s.materials[0].sheen_color = [float("inf"), 1.0, 1.0]
    s.materials[0].sheen = 0.0
    img, ref = both(oracle_lib, gpu, s, 33, 33, 2)
    check(img, ref, "infinite sheen colour")


# Free paths from far below the boundary rays' minimum distance to far above
# the object: exits on the first step, on a later one, at the step limit, and
# walks whose boundary ray escapes through an open sheet.
@pytest.mark.parametrize("scale", [0.0, 0.02, 0.3, 50.0])
@pytest.mark.parametrize("closed", [True, False])
def test_subsurface_walks(oracle_lib, gpu, scale, closed):
    wl = workloads.closed_box(40, 40)
    scene = wl.scene if closed else R.mesh_light_scene(0.0)
    for m in scene.materials:
        m.subsurface = 1.0
        m.subsurface_scale = scale
        m.subsurface_color = [0.9, 0.5, 0.3]
    if not closed:
        scene.lights = R.analytic_lights()[1:2]
    img, ref = both(oracle_lib, gpu, scene, 40, 40, 4, camera=wl.camera if closed else None)
    check(img, ref, f"walks {scale} closed {closed}")


@pytest.mark.parametrize("deferred", [True, False])
def test_lanes_that_part(oracle_lib, gpu, deferred):
    """Dispersion, scattering media and coloured translucency part the lanes of a
    group; with sorted hits the entries of both kernels go in material order."""
    wl = R.fuzz_box(3)
    scene = wl.scene
    m = scene.materials[0]
    m.transmission, m.metalness, m.thin_walled = 1.0, 0.0, False
    m.transmission_dispersion_scale, m.transmission_dispersion_abbe_number = 1.0, 9.0
    with PathTracer(0) as t:
        t.set_tuning(sort_hits=1 if deferred else 0)
        t.set_scene(scene)
        img = t.render(wl.camera, 41, 39, 0, 8, 4)
    o = oracle_lib.OracleTracer()
    o.set_scene(scene)
    check(img, o.render(wl.camera, 41, 39, 0, 8, 4), "parting lanes")
