"""The engine's host-side memory handling when an allocation fails, on a stub
runtime (tests/cpp/alloc_failures.cpp): no GPU runs out of memory for it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_alloc_failures(tmp_path):
    exe = str(tmp_path / "alloc_failures")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-Wall", "-Wextra",
                    "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "reyn_b200", "csrc"),
                    "-isystem", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "alloc_failures.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
