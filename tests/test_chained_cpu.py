"""Chained kernels (csrc/launch.h) start while the kernel before them runs, so
nothing they read is read-only for their whole life, which is what a
__restrict__ parameter lets the compiler assume."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "cl-ops_gb300" / "csrc"


def _kernels():
    """(file, name, parameters, body) of the __global__ functions."""
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = f.read_text()
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)"
                             r"\s*)?(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield f.name, m[1], m[2], text[m.end():i]


def test_chained_kernels_take_no_restrict_parameters():
    chained = [(f, k, p) for f, k, p, body in _kernels() if "pdl_wait()" in body]
    assert len(chained) >= 20
    assert not [(f, k) for f, k, p in chained if "__restrict__" in p]
