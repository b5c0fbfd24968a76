"""Which levels of an AMG setup are aggregated on the device (the C library's rules, compiled and run as
a host program)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_aggregation_rule(tmp_path):
    exe = str(tmp_path / "test_aggregation_rule")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "cfd_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_aggregation_rule.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
