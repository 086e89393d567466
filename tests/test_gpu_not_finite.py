"""Values that are not finite and meet a zero weight: zero times infinity is
not zero, so terms with a weight of zero are left out only where their other
factors are finite. Against the oracle, which leaves nothing out; tolerance as
in test_gpu_path_groups.py."""
import pytest

import ref_scenes as R
from hdcodex_b200 import PathTracer
from hdcodex_b200.scene import DOME
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


@pytest.mark.parametrize("factor", [INF, -INF, NAN])
@pytest.mark.parametrize("kind", [1, 2], ids=["analytic", "with dome"])
def test_diffuse_factor_of_a_light(oracle_lib, factor, kind):
    """Materials without layered lobes: the specialised closure, if all is finite."""
    s = R.mesh_light_scene(0.0)
    s.lights = R.analytic_lights()[:2]
    if kind == 2:
        s.lights.append(s.lights[0].copy(id="/dome", type=DOME, color=[0.3, 0.4, 0.5], texture=""))
    s.lights[1].diffuse = factor
    compare(oracle_lib, s, f"diffuse factor {factor}")
