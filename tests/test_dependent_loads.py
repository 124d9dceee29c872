"""Dependent launches (azk_internal.h): a kernel that is set up while the kernel ahead
of it still writes must not read that kernel's output as read-only data.  So in the
sources every __ldg and every `const T* __restrict__` parameter of such a kernel names
data that copies or completed set-up work wrote; everything else goes through
ld_written or __ldcg."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apple_b200", "csrc")
FILES = ["circle_kernels.cu", "fft_m31_kernels.cu", "merkle_kernels.cu", "witness_fft.cu"]

# First names of what a __ldg may read, by file: domain tables and inverse layers
# (src, p, inv, job.inv), roots and transforms of fixed sequences (roots, kf), raw
# messages (raw, p), job records (from), and the inputs of kernels that are launched
# plainly (in, prev of fold_kernel and fold_qm31_inv_kernel).
READ_ONLY = {
    "circle_kernels.cu": {"src", "inv", "in", "job.inv"},
    "fft_m31_kernels.cu": {"p"},
    "merkle_kernels.cu": {"job.inv", "p", "from"},
    "witness_fft.cu": {"roots", "kf"},
}
PLAIN_KERNEL_INPUTS = {"fold_kernel": {"job.prev"}, "fold_qm31_inv_kernel": {"prev"}}
READ_ONLY_PARAMETERS = {"jobs", "work", "inst", "ids", "inv_words", "roots"}


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
    return re.sub(r"__launch_bounds__\([^)]*\)", "", text)


def call_arguments(text, start):
    """The text between the parenthesis at `start` and its match."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "(") - (text[i] == ")")
        if depth == 0:
            return text[start + 1:i]
    raise AssertionError("unbalanced parentheses")


def function_at(text, pos):
    """Name of the kernel or device function whose body holds `pos`."""
    last = None
    for m in re.finditer(r"\b(\w+)\s*\([^;{}]*\)\s*\{", text[:pos]):
        if m.group(1) not in ("if", "for", "while", "switch", "constexpr"):
            last = m.group(1)
    return last


@pytest.mark.parametrize("name", FILES)
def test_read_only_loads_name_read_only_data(name):
    text = source(name)
    bad = []
    for m in re.finditer(r"\b__ldg\(", text):
        arg = call_arguments(text, m.end() - 1)
        arg = re.sub(r"(reinterpret_cast|static_cast)<[^>]*>\s*", "", arg).replace("(", " ").strip()
        base = re.match(r"[\w.]+", arg).group(0)
        if base in READ_ONLY[name] or base in PLAIN_KERNEL_INPUTS.get(function_at(text, m.start()), ()):
            continue
        bad.append((function_at(text, m.start()), arg))
    assert not bad, bad


def test_dependent_kernels_take_no_restricted_inputs_but_tables():
    seen = set()
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        text = source(name)
        for m in re.finditer(r"\blaunch_dependent\(\s*(\w+)", text):
            kernel = m.group(1)
            if kernel == "void":
                continue
            seen.add(kernel)
            d = re.search(r"__global__[^;{]*?\b" + kernel + r"\s*\(", text)
            assert d, kernel
            params = call_arguments(text, d.end() - 1)
            names = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)
            assert set(names) <= READ_ONLY_PARAMETERS, (kernel, names)
            body = text[d.end():]
            assert "dependent_begin()" in body[:body.find("__global__") if "__global__" in body else len(body)], kernel
    assert len(seen) >= 10, seen
