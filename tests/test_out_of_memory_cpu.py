"""Entry points that cannot allocate return an error, without a GPU."""
import os
import subprocess

from fbgemm_b200 import _capi, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_allocations_are_return_codes(tmp_path):
    _capi.lib()
    exe = str(tmp_path / "out_of_memory_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", build.INCLUDE,
                    os.path.join(ROOT, "tests", "cpp", "out_of_memory_test.cc"), "-o", exe, "-L", build.PKG_DIR,
                    "-lfbgemm_b200", "-Wl,-rpath," + build.PKG_DIR], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
