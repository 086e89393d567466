"""The bound of an automatic wave by device memory (hdcodex_b200/csrc/wave_plan.h):
host-only C++, compiled and run here with g++; and, on a GPU, that path state
takes the bytes per path that the bound counts."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_automatic_waves_fit_the_memory(tmp_path):
    exe = tmp_path / "wave_plan_tests"
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "hdcodex_b200", "csrc"),
                            os.path.join(ROOT, "tests", "cpp", "wave_plan_tests.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "all wave plan checks passed" in run.stdout, run.stdout + run.stderr


@pytest.mark.gpu
def test_path_state_takes_the_bytes_that_are_counted(tmp_path):
    from hdcodex_b200 import PathTracer, workloads
    from hdcodex_b200.tracer import device_memory_usage
    src = tmp_path / "bytes.cpp"
    src.write_text('#include "wave_plan.h"\n#include <cstdio>\nint main() { std::printf("%d", static_cast<int>(hdcx::kPathStateBytes)); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "hdcodex_b200", "csrc"), str(src), "-o", str(tmp_path / "bytes")], check=True)
    counted = int(subprocess.run([str(tmp_path / "bytes")], capture_output=True, text=True, check=True).stdout)
    header = open(os.path.join(ROOT, "include", "hdcx.h")).read()
    assert {int(n) for n in re.findall(r"about (\d+) bytes per path", header)} == {counted}
    wl = workloads.closed_box(width=256, height=256)
    paths = 256 * 256 * 3  # a sample
    used = []
    with PathTracer(0) as t:
        t.set_scene(wl.scene)
        for samples in (20, 40):
            t.set_wave_size(samples * paths)
            t.render(wl.camera, 256, 256, 0, 1, 40)
            used.append(device_memory_usage(0)[0])
    # Rounding up to whole groups and their bytes: below one byte a path.
    assert counted - 1 < (used[1] - used[0]) / (20 * paths) <= counted
