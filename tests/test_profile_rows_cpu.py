"""Which unit of t reads a row of the row-sum profiles (wrt-project_b200/csrc/
profile_dev.cuh): exactly one, compiled here on the CPU with and without fused
multiply-adds."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("contract", ["off", "fast"])
def test_every_row_is_in_one_unit(tmp_path, contract):
    exe = tmp_path / "profile_rows_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-ffp-contract={contract}",
                    str(HERE / "profile_rows_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
