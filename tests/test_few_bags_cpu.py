"""Which lookups go to the kernel for a handful of bags, without a GPU."""
import os
import subprocess

from fbgemm_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rule_of_few_bags(tmp_path):
    exe = str(tmp_path / "few_bags_rule_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "few_bags_rule_test.cc"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
