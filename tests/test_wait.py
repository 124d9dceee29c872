"""The library's waits, compiled for the host: how many threads may spin, and when the
others sleep; and the turns of large uploads."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_waits(tmp_path):
    exe = tmp_path / "wait_check"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "apple_b200", "csrc"), os.path.join(ROOT, "tests", "wait_check.cpp"),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
