"""The message readers of the hash and raw-leaf kernels, compiled for the host: the
words of messages of 0 to 136 bytes at every alignment, with no load outside the
message (a buffer may end with its last message, and its neighbours may be written
meanwhile)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_readers_stay_inside_the_message(tmp_path):
    exe = tmp_path / "message_reader_check"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "apple_b200", "csrc"), os.path.join(ROOT, "tests", "message_reader_check.cpp"),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert "message readers ok" in r.stdout
