"""Kernels that are set up while the one before them still writes: nothing they read is promised to the compiler as constant
for their whole run (a load through such a promise is not ordered by grid_dependency_wait)."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rbf_attention_b200", "csrc")


def _kernels(source):
    """(name, parameters, body) of the kernels defined in a source file."""
    for m in re.finditer(r"__global__ void\s+__launch_bounds__\(", source):
        depth, at = 1, m.end()
        while depth:                                    # the launch bounds may hold parentheses of their own
            depth += {"(": 1, ")": -1}.get(source[at], 0)
            at += 1
        name = re.match(r"\s*(\w+)\(", source[at:])
        start = at + name.end()
        end = source.index(") {", start)
        depth, stop = 1, end + 3
        while depth:
            depth += {"{": 1, "}": -1}.get(source[stop], 0)
            stop += 1
        yield name.group(1), source[start:end], source[end:stop]


@pytest.mark.parametrize("file", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_inputs_of_dependent_kernels_are_not_promised_constant(file):
    with open(os.path.join(CSRC, file)) as f:
        source = f.read()
    launched = set(re.findall(r"launch_dependent\(\s*(\w+)", source))
    waiting = {name for name, _, body in _kernels(source) if "grid_dependency_wait()" in body}
    assert len(waiting) >= len(launched)
    for name, parameters, _ in _kernels(source):
        if name in waiting:
            promised = [p for p in parameters.split(",") if "__restrict__" in p and re.match(r"\s*const\b", p)]
            assert not promised, (name, promised)
