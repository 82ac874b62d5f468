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


def body_of(name, kernel):
    with open(os.path.join(CSRC, name)) as f:
        found = [body for signature, body in functions(f.read()) if re.search(r"\b%s\(" % kernel, signature)]
    assert len(found) == 1
    return found[0]


def triggers_after_wait(body, chained):
    """Whether a kernel lets its successor start only once its own wait is over (calls under `if (chained)` or `if (!chained)`
    count in the one case or the other)."""
    events = re.findall(r"(?:if \((!?chained)\) )?(pdl_launch_dependents|pdl_wait)\(\)", body)
    order = [call for condition, call in events if condition in ("", "chained" if chained else "!chained")]
    assert sorted(order) == ["pdl_launch_dependents", "pdl_wait"]
    return order[0] == "pdl_wait"


@pytest.mark.parametrize("exchange", ["k_reduce_rows", "k_reduce_exchange_update"])
@pytest.mark.parametrize("empty_first_steps", [0, 2])
def test_early_image_copies_follow_whatever_wrote_the_images(exchange, empty_first_steps):
    """In a training loop the gradient kernel of a later step copies its first images before its wait.  A kernel may start when the
    one before it has triggered, which says that the launches further back are complete only if that trigger came after a
    wait; the kernel that wrote the images (launch 0, which may trigger as early as it likes) has to be among them."""
    grad = body_of("fused_train.cu", "k_grad_partials")
    reduce_after = triggers_after_wait(body_of("fused_train.cu" if exchange == "k_reduce_rows" else "dp_exchange.cu", exchange), False)
    launches, trained = [("writer", False, False)], False
    for step in range(empty_first_steps + 4):
        if step >= empty_first_steps:          # (a rank without images of a global batch launches no gradient kernel)
            launches.append(("grad", trained, triggers_after_wait(grad, trained)))
            trained = True
        launches.append(("reduce", False, reduce_after))
    complete = -1                              # launches up to this one are complete when launch i starts
    for i, (kind, chained, _) in enumerate(launches):
        if i > 0 and launches[i - 1][2]:
            complete = max(complete, i - 2)
        assert not (kind == "grad" and chained) or complete >= 0, i
    assert re.search(r"first > 0 \|\| e > 0|trained", open(os.path.join(CSRC, "fused_train.cu")).read())
    assert re.search(r"stream, trained\);.*?trained = trained \|\| hi > lo;", open(os.path.join(CSRC, "dp_exchange.cu")).read(), re.S)
