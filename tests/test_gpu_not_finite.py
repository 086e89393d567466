"""Values that are not finite and meet a zero weight: zero times infinity is
not zero, so terms with a weight of zero are left out only where their other
factors are finite. Against the oracle, which leaves nothing out; tolerance as
in test_gpu_path_groups.py."""
import pytest

import ref_scenes as R
from hdcodex_b200 import PathTracer
from test_gpu_path_groups import check

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def compare(oracle_lib, scene, what):
    o = oracle_lib.OracleTracer()
    o.set_scene(scene)
    ref = o.render(R.base_camera(), 37, 29, 0, 8, 4)
    with PathTracer(0) as t:
        t.set_scene(scene)
        check(t.render(R.base_camera(), 37, 29, 0, 8, 4), ref, what)


def receiver(mesh_light, lights):
    s = R.mesh_light_scene(1.0 if mesh_light else 0.0)
    s.lights = R.analytic_lights()[1:3] if lights else []
    s.materials[0].coat = 0.3  # the whole closure
    return s


@pytest.mark.parametrize("color", [[NAN, 0.5, 0.5], [0.5, INF, 0.5], [0.2, 0.2, -INF]], ids=["nan", "inf", "-inf"])
@pytest.mark.parametrize("mesh_light,lights", [(False, True), (True, True), (True, False), (False, False)])
def test_translucent_colour_without_weight(oracle_lib, color, mesh_light, lights):
    s = receiver(mesh_light, lights)
    for m in s.materials:
        m.translucent_weight, m.translucent_color = 0.0, color
    compare(oracle_lib, s, f"translucent colour {color}")
