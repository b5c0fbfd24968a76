"""Order of the records by which the host follows a solve, over the wrap of their number (the C
library's rule, compiled and run as a host program)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_progress_rule(tmp_path):
    exe = str(tmp_path / "test_progress_rule")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "cfd_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_progress_rule.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
