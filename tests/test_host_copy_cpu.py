"""The threaded copies between a caller's arrays and page-locked memory, without
a GPU: compiled with their own small driver."""
import os
import subprocess

import pytest

from fbgemm_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_copy") / "host_copy_test")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "host_copy_test.cc"), os.path.join(build.CSRC, "host_copy.cc"),
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", [
    "exact",   # every byte arrives; a copy that ends early leaves nothing behind
    "fork",    # a forked child copies alone and ends
    "idle",    # waiting for a transfer keeps no core busy
    "again",   # helpers that left for want of work come back
])
def test_copies(driver, what):
    res = subprocess.run([driver, what], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
