"""The rule that chooses the occlusion kernel of a launch (csrc/occlusion_choice.h),
compiled and checked on the CPU; test_gpu_fetch_kernel.py compares the pictures."""
import subprocess
from pathlib import Path

import pytest

from umbreon_gb300 import scenes

ROOT = Path(__file__).resolve().parent.parent


def test_occlusion_choice(tmp_path):
    exe = tmp_path / "test_occlusion_choice"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(ROOT / "umbreon_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_occlusion_choice.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("make,lights", [
    (lambda: scenes.space_filling(n=50, width=8, height=8), 1),
    (lambda: scenes.ball_and_stick(n=50, width=8, height=8, supersample=1, ao_samples=16), 2)])
def test_compared_launches_have_these_rays(make, lights):
    """The shadow rays per hit that the launches of the C++ test count."""
    sc, _ = make()
    assert len(sc.lights) == lights and all(light.angularRadius == 0.0 for light in sc.lights)
