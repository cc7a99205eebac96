"""The walk over a vertex's arcs by its lanes (cgc_arcs.h), on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranges_up_to_the_largest_arc_ids(tmp_path):
    exe = str(tmp_path / "test_arc_walk")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(ROOT, "cugip_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "test_arc_walk.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and "arc walk ok" in out.stdout, out.stdout + out.stderr
