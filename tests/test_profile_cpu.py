"""The geometry of the row-sum profiles (wrt-project_b200/csrc/profile_dev.cuh) is
plain scalar code: compiled here on the CPU and summed up as the kernel sums it,
against direct sums over the lattice rows (every class of phi, both samplers,
lattices shorter and longer than the cube), with every index checked."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_pieces_match_direct_sums(tmp_path):
    exe = tmp_path / "profile_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    str(HERE / "profile_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_merged_knots_match_the_splines(tmp_path):
    """csrc/backproj_dev.cuh: the merged spline of all latitudes against the
    splines themselves."""
    exe = tmp_path / "backproj_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    str(HERE / "backproj_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
