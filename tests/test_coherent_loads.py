"""Kernels that become resident beside the launch in front of them read its results by plain loads (source check, no GPU)."""

import glob
import os
import re

from freetoken_b200.csrc import build


def functions(text):
    """Every function with a body: its head and the body, comments taken out."""
    text = re.sub(r"//.*", "", text)
    for m in re.finditer(r"(?:__global__|__device__)[^;{}]*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(), text[m.end():at]


def violations(text):
    found = []
    for head, body in functions(text):
        if "pdl_wait" not in body and "__device__" not in head:
            continue                                      # launched behind whatever is in front of it
        name = ([n for n in re.findall(r"(\w+)\s*\(", head) if n != "__launch_bounds__"] + [head])[0]
        if re.search(r"const [\w ]+\*\s*__restrict__", head):
            found.append((name, "a const __restrict__ parameter"))
        if "__ldg(" in body or "ld.global.nc" in body:
            found.append((name, "a read-only load"))
    return found


def test_kernels_launched_early_read_by_plain_loads():
    files = glob.glob(os.path.join(build.HERE, "*.cu")) + glob.glob(os.path.join(build.HERE, "*.cuh"))
    waiting = 0
    for path in files:
        with open(path) as f:
            text = f.read()
        assert violations(text) == [], os.path.basename(path)
        waiting += sum("pdl_wait" in body for head, body in functions(text) if "__global__" in head)
    assert waiting > 50


def test_the_check_finds_both_forms():
    kernel = "template <typename T>\n__global__ void __launch_bounds__(32 * (A < 8 ? A : 8)) k(const T%s x, T* __restrict__ y) {\n pdl_wait();\n y[0] = %s; if (y) { y[1] = 0; }\n}\n"
    assert violations(kernel % ("*", "x[0]")) == []
    assert violations(kernel % ("* __restrict__", "x[0]")) == [("k", "a const __restrict__ parameter")]
    assert violations(kernel % ("*", "__ldg(x)")) == [("k", "a read-only load")]
    assert violations((kernel % ("* __restrict__", "__ldg(x)")).replace("pdl_wait", "other")) == []
