"""The triangle test's double-precision redo: both forms give the same bits (CPU)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_triangle_redo(tmp_path):
    from umbreon_gb300 import build
    cuda = Path(build._nvcc()).resolve().parent.parent
    exe = tmp_path / "test_triangle_redo"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(cuda / "include"),
                        "-I", str(ROOT / "include"), "-I", str(ROOT / "umbreon_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_triangle_redo.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
