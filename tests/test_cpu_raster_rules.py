"""The kernels' shortcuts against the rules they stand for (host build of their headers)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shortcuts(tmp_path):
    """No row before walk_first_late_row is late (every width <= 800, top row < 600; run with
    3840 2160 the program covers the whole range), box_bounds encloses every
    pixel's depth, tight_box and row_span leave no covered pixel out, ssao_tap counts as ssao_count
    does, and the shadow bias and limits hold."""
    exe = tmp_path / "rrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "openclrenderer_gb300", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "raster_rules_check.cpp")], check=True)
    r = subprocess.run([str(exe), "800", "600", "200000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_walk_skip_rows(tmp_path):
    """The rasterisers' bits of skipped rows are walk_visits' rows."""
    exe = tmp_path / "wsc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "openclrenderer_gb300", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "walk_skip_check.cpp")], check=True)
    r = subprocess.run([str(exe), "3", "3000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_span_slack(tmp_path):
    """Spans of triangles with vertices off the surface leave no covered pixel out."""
    exe = tmp_path / "ssc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "openclrenderer_gb300", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "span_slack_check.cpp")], check=True)
    r = subprocess.run([str(exe), "5", "200000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
