"""Kernels that start beside the one in front of them (programmatic dependent launches): what they declare as constant
has to be constant for as long as they run, so only the caller's arrays may be read that way.  Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chunkedgreedy_b200", "csrc")
CALLERS = {"ptr", "ind", "ptr_old", "new_order"}  # arrays no kernel of a call writes


def _kernels():
    """(file, name, parameters, body) of every kernel"""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\((?:[^()]|\([^()]*\))*\)\s*)*(\w+)\s*\(", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params = text[m.end():at - 1]
            start = text.index("{", at)
            depth, at = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield name, m.group(1), params, text[start:at]


KERNELS = list(_kernels())
DEPENDENT = [k for k in KERNELS if "wait_for_kernels_before" in k[3]]


def test_kernels_are_found():
    names = {k[1] for k in DEPENDENT}
    assert {"ptr_new_kernel", "row_list_kernel", "compact_kernel", "heavy_rounds_kernel", "apply_flat_kernel"} <= names


@pytest.mark.parametrize("kernel", DEPENDENT, ids=lambda k: k[1])
def test_constant_arrays_are_the_callers(kernel):
    _, _, params, body = kernel
    constant = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)
    constant += re.findall(r"__ldg\(\s*(?:a\.)?(\w+)", body)
    assert set(constant) <= CALLERS


def test_every_kernel_launched_that_way_waits():
    waiting = {k[1] for k in DEPENDENT}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            text = open(os.path.join(CSRC, name)).read()
            launched = re.findall(r"launch_behind\([^;]*?(\w+_kernel)\b", text)
            assert set(launched) <= waiting, name
