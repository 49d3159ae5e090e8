"""Kernels are launched with programmatic stream serialisation, so each has to
wait for the kernel before it: grid_entry() as its first statement."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "horsepower_gb300", "csrc")


def kernels(text):
    """(name, first statement) of every kernel definition in a source text."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*(\((?:[^()]|\([^()]*\))*\))\s*)?(\w+)\s*\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        body = re.match(r"\s*\{\s*([^;]*;)", text[k:])
        if body:
            yield m.group(2), body.group(1)


def test_every_kernel_waits_first():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = open(path).read()
        for name, first in kernels(text):
            if name == "chain_kernel":
                continue
            seen += 1
            assert first == "grid_entry();", (os.path.basename(path), name, first)
    assert seen > 150


def test_generated_kernels_wait():
    """The chain compiler's kernels hold the same wait (one per kernel text)."""
    text = open(os.path.join(CSRC, "k_fused.cu")).read()
    assert text.count("__global__ void __launch_bounds__(256) chain_kernel(") == text.count("griddepcontrol.wait") == 2
