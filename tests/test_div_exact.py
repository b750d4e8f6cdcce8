"""The division by a known reciprocal that the generate launch uses for
positions in voxel units equals IEEE division."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_div_matches_ieee_division(tmp_path):
    exe = str(tmp_path / "div_check")
    src = os.path.join(REPO, "tests", "div_check.cpp")
    inc = os.path.join(REPO, "marching_cube_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", inc, src, "-o", exe, "-lm"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "0 mismatches" in r.stdout, r.stdout
