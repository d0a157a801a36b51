"""Kernels that may be resident before their inputs are written (they begin with griddepcontrol.wait) read them with
plain loads: nothing but that keeps a load behind the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vulkanforge_b200", "csrc")


def _kernels():
    """(file, name, text from its parameters to the end of its body) of every __global__ function."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__", text):
            kernel = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", lambda b: " " * len(b.group()), text[m.end():m.end() + 600]))
            at, depth = text.index("{", m.end() + kernel.end()), 0
            for end in range(at, len(text)):
                depth += (text[end] == "{") - (text[end] == "}")
                if depth == 0:
                    break
            yield name, kernel.group(1), text[m.end() + kernel.start():end]


def test_no_read_only_loads_behind_a_dependent_launch():
    waiting = [k for k in _kernels() if "pdl_wait()" in k[2] or "griddepcontrol.wait" in k[2]]
    assert len(waiting) >= 16                              # the scan finds them
    bad = [(f, k) for f, k, text in waiting if "__ldg" in text or "__restrict__" in text]
    assert not bad
