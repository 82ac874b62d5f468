"""Kernels that may start while their predecessor still runs (programmatic dependent launch, pdl_wait) must not read global memory
through the read-only path: PTX promises ld.global.nc only for data that nobody writes during the kernel's lifetime, and the
compiler may move such loads in front of the wait.  In the source that is __ldg, and a `const T* __restrict__` parameter."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "high-performance-cnn-framework-using-cuda_b200", "csrc")
FILES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*")))
READ_ONLY = re.compile(r"__ldg\s*\(|ld\.global\.(?:\w+\.)*nc")
READ_ONLY_PARAMETER = re.compile(r"const\s+\w[\w:]*\s*\*\s*__restrict__\s*\w+")


def functions(text):
    """(signature, body) of every device function and kernel of a source."""
    text = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
    for m in re.finditer(r"__(?:global|device)__[^;{}]*?\w+\s*\([^;{}]*\)\s*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(0), text[m.end():at]


def offences(text):
    for signature, body in functions(text):
        kernel = "__global__" in signature
        if kernel and "pdl_wait(" not in body:      # an ordinary launch begins when its predecessor is complete
            continue
        name = re.search(r"(\w+)\s*\([^()]*(?:\([^()]*\)[^()]*)*\)\s*\{$", signature)
        for what in READ_ONLY.findall(body) + READ_ONLY_PARAMETER.findall(signature):
            yield "%s: %s" % (name.group(1) if name else signature[:60], what)


def test_the_check_finds_what_it_looks_for():
    kernel = "__global__ void __launch_bounds__(32)\nk_x(%s p, int* __restrict__ q) { %s q[0] = %s; }"
    assert list(offences(kernel % ("const int* __restrict__", "pdl_wait();", "p[0]"))) == ["k_x: const int* __restrict__ p"]
    assert list(offences(kernel % ("const int*", "pdl_wait();", "__ldg(p)"))) == ["k_x: __ldg("]
    assert not list(offences(kernel % ("const int*", "pdl_wait();", "p[0]")))
    assert not list(offences(kernel % ("const int* __restrict__", "", "p[0]")))


@pytest.mark.parametrize("name", FILES)
def test_no_read_only_loads_beside_a_running_predecessor(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    if "pdl_wait(" not in text and name.endswith(".cu"):
        return
    assert not list(offences(text))
