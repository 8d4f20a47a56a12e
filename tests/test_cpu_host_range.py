"""Which host buffers the kernels write directly, on made-up allocations (host build of the rule)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_mapped_range(tmp_path):
    exe = tmp_path / "hrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "openclrenderer_gb300", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "host_range_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
