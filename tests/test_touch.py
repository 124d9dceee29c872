"""The page touch ahead of large downloads, compiled for the host: running out of memory
while it starts its threads must not end the process."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_touch_survives_failed_allocations(tmp_path):
    exe = tmp_path / "touch_check"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "apple_b200", "csrc"), os.path.join(ROOT, "tests", "touch_check.cpp"),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)
    assert "touch ok" in r.stdout
