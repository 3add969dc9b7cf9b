"""Kernels that start before the kernel in front of them has ended (they wait in griddepcontrol.wait) must not read what that kernel writes
through the read-only path: __ldg, or a load the compiler turns into one because the pointer is const __restrict__, is defined only for
memory that stays constant while the kernel runs, and may be moved in front of the wait.  Checked on the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "slai_b200", "csrc")
CONSTANT = {"norm_w", "gamma", "beta", "theta", "table", "qdata", "tokens"}  # weights, tables, a prompt's ids (copied before any launch)
CONSTANT_LOADS = CONSTANT | {"w4p", "b4p"}  # norm weights and biases as vectors of four
WAIT = "griddepcontrol.wait"


def functions(text):
    """(qualifier, parameters, body) of every __global__ or __device__ function."""
    for m in re.finditer(r"__(global|device)__", text):
        at = text.find("(", m.end())
        bounds = text.find("__launch_bounds__", m.end(), at)
        if bounds >= 0:
            at = text.find("(", text.find(")", at) + 1)
        depth, i = 0, at
        while True:  # parameters
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        params, brace = text[at:i], text.find("{", i)
        if text[i:brace].strip():
            continue  # a declaration
        depth, j = 0, brace
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        yield m.group(1), params, text[brace:j]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_no_read_only_loads_of_what_a_predecessor_writes(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    file_waits = WAIT in text
    for kind, params, body in functions(text):
        if WAIT in body or (kind == "device" and file_waits):  # helpers are inlined into the kernels of the file
            for p in params.split(","):
                if "__restrict__" in p:
                    assert re.findall(r"\w+", p)[-1] in CONSTANT, (os.path.basename(path), p.strip())
            for load in re.findall(r"__ldg\(([^;]*)", body):
                assert CONSTANT_LOADS & set(re.findall(r"\w+", load)), (os.path.basename(path), load.strip())
