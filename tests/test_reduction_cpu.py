"""Positions along a line of the staged reduction (wrt-project_b200/csrc/
reduction_dev.cuh), compiled here on the CPU: the cells that the kernel reads stay
inside its staged arrays for every number of layers it accepts."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("contract", ["off", "fast"])
def test_positions_stay_inside(tmp_path, contract):
    exe = tmp_path / "reduction_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-ffp-contract={contract}",
                    str(HERE / "reduction_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
