"""Which of the caller's device planes a frame is written to directly: the host
rule (csrc/frame_planes.h), compiled and checked on the CPU."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_frame_planes(tmp_path):
    exe = tmp_path / "test_frame_planes"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(ROOT / "umbreon_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_frame_planes.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
