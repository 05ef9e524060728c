"""A context's device memory (csrc/context.cu) on the CPU, against a fake of the
CUDA runtime's allocations."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_context_memory(tmp_path):
    from umbreon_gb300 import build
    cuda = Path(build._nvcc()).resolve().parent.parent
    exe = tmp_path / "test_context_memory"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(cuda / "include"), "-I", str(ROOT / "include"),
                        "-I", str(ROOT / "umbreon_gb300" / "csrc"), "-I", str(ROOT / "tests" / "cpp"),
                        str(ROOT / "tests" / "cpp" / "test_context_memory.cpp"), "-x", "c++",
                        str(ROOT / "umbreon_gb300" / "csrc" / "context.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
