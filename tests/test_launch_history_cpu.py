"""What a context knows of the launches beside one, without a GPU."""
import os
import subprocess

from fbgemm_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launches_on_other_streams_are_counted(tmp_path):
    exe = str(tmp_path / "launch_history_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "launch_history_test.cc"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
