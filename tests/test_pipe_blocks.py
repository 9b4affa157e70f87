"""The block order of the pipelined FP64 moments + Poisson launch, on CPU: on any number of SMs
every block that waits is preceded by one that ends its wait (tests/native/pipe_blocks_check.cpp).
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_every_wait_ends_on_any_number_of_sms(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "pipe_blocks_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(ROOT / "veritas_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "pipe_blocks_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert "grids end" in r.stdout
