"""Size rules of the host code, compiled and run without a GPU."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_rules(tmp_path):
    exe = str(tmp_path / "rules")
    cmd = ["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ursa_b200", "csrc"),
           os.path.join(ROOT, "tests", "cpp", "test_host_rules.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout
