"""CPU test of the allocation-free entry point's wait records: the host code that chooses them, compiled for a model of the GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_every_call_starts_clear_and_the_last_one_is_seen(tmp_path):
    exe = tmp_path / "wait_records_selftest"
    src = os.path.join(ROOT, "tests", "host", "wait_records_selftest.cpp")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-o", str(exe), src])
    assert "wait records ok" in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
