"""Hash and transcript forms that only the kernels run, compiled for the host and
compared with the CPU oracle."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_device_forms_on_host(tmp_path):
    exe = tmp_path / "device_forms_check"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-fopenmp", "-I", os.path.join(ROOT, "oracle"), "-I", os.path.join(ROOT, "apple_b200", "csrc"),
                        os.path.join(ROOT, "tests", "device_forms_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert "device forms ok" in r.stdout
