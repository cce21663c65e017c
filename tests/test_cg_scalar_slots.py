"""The CG kernels hand each other scalars through device slots.  Nothing orders the blocks of one launch,
so a slot that a kernel stores must not be read by its other threads (an early return on such a value
would also split a block ahead of its barriers).  Checked on the source, where it does not depend on timing."""
import os
import re

import pytest

from conftest import ROOT

SRC = open(os.path.join(ROOT, "sod2d_refmap_b200", "csrc", "sod_cg.cu")).read()


def kernel_body(name):
    start = SRC.index("{", SRC.index(" " + name + "("))
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(SRC[i], 0)
        i += 1
        if depth == 0:
            return re.sub(r"//[^\n]*", "", SRC[start:i])


ONE = r"if \(blockIdx\.x == 0 && threadIdx\.x == 0\) (\{[^{}]*\}|[^;{}]*;)"
STORE = r"scal\[(S_\w+)\]\s*[+\-*/]?=(?!=)"


def accesses(body):
    """(slots read by every thread, slots stored by one thread)."""
    rest = re.sub(ONE, "", body)
    one = "".join(re.findall(ONE, body))
    assert not re.findall(STORE, rest), "a scalar slot stored by more than one thread"
    return set(re.findall(r"scal\[(S_\w+)\]", rest)), set(re.findall(STORE, one))


@pytest.mark.parametrize("name", ["k_lap_elem", "k_lap_elem_async", "k_lap_gather", "k_cg_update", "k_cg_pupdate"])
def test_no_slot_is_read_and_stored_in_one_launch(name):
    read, stored = accesses(kernel_body(name))
    assert read, name  # each of them tests for the end of the solve
    assert not read & stored, (name, read & stored)
