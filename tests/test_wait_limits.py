"""What the tensor-core kernels do when a bounded wait runs out, read from the
source (a wait that runs out is not brought about on the device)."""
import os
import re

import pytest

from test_cluster_order import CSRC, kernels


def bodies():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            with open(os.path.join(CSRC, f)) as fh:
                out += [(n, b) for n, b in kernels(fh.read()) if "mbar_wait" in b]
    return out


def open_blocks(body, at):
    """Headers of the blocks around position `at`."""
    stack, start = [], 0
    for i, ch in enumerate(body[:at]):
        if ch == "{":
            stack.append(body[start:i].strip())
        elif ch == "}":
            stack.pop()
        if ch in "{};":
            start = i + 1
    return stack


@pytest.mark.parametrize("name,body", bodies(), ids=lambda v: v if "\n" not in v else "body")
def test_warps_agree_on_a_wait(name, body):
    """A wait by a whole warp is voted on: lanes that leave alone would be
    missing from the warp's next .aligned instruction.  Single threads may
    wait by themselves."""
    waits = [m.start() for m in re.finditer(r"\bmbar_wait\(", body)]
    assert waits
    for at in waits:
        assert any(re.search(r"\(ln == 0\)|\(tid == 0\)", h) for h in open_blocks(body, at)), (name, body[at:at + 60])


def test_a_bad_pivot_does_not_hide_it():
    """The error word of the dense factorisation is -1 after a wait that ran
    out, reported as such; a panel number is only put where it was 0.  Every
    unconditional store into an error word is the -1."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                for value in re.findall(r"atomicExch\((?:\w+[.>-]+)?err,\s*(.*)\);", fh.read()):
                    assert value == "-1", (f, value)
