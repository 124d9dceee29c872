"""Importing the package leaves the process's shared ctypes objects as they were, and
its own prototype makes bytes objects to fill."""
import subprocess
import sys


def test_import_leaves_pythonapi_alone():
    code = """
import ctypes
f = ctypes.pythonapi.PyBytes_FromStringAndSize
before = (f.restype, f.argtypes)
import apple_b200
from apple_b200 import plans
assert ctypes.pythonapi.PyBytes_FromStringAndSize is f and (f.restype, f.argtypes) == before, (f.restype, f.argtypes)
b, at = plans._fresh_bytes(5)
ctypes.memmove(at, b"abcde", 5)
assert b == b"abcde" and type(b) is bytes
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)
