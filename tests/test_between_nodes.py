"""The cells and sides for which generate takes a vertex's voxel and its normal's
samples to lie beside the vertex's edge: they do, over random edges, distances
and cells, and for the cells and sides left out they do not."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_between_nodes(tmp_path):
    exe = str(tmp_path / "between_check")
    src = os.path.join(REPO, "tests", "between_check.cpp")
    inc = os.path.join(REPO, "marching_cube_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, src, "-o", exe, "-lm"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
