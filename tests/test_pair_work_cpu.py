"""CPU test of the CTA-pair GEMM's work split: the device header's own code, compiled for the host."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_every_k_tile_of_every_tile_has_one_unit(tmp_path):
    exe = tmp_path / "pair_work_selftest"
    src = os.path.join(ROOT, "tests", "host", "pair_work_selftest.cu")
    subprocess.check_call(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe), src])
    assert "pair work ok" in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
