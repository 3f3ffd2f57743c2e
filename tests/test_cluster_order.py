"""A CTA may use another CTA's shared memory only once that CTA is known to
run: in every kernel that maps a peer's shared memory, a barrier of the
cluster stands before the first mapping, outside any loop or condition.  Read
from the source, as a store into a CTA that has not started is not to be run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "millepede-ii_gb300", "csrc")


def kernels(text):
    """(name, body) of the __global__ functions, comments removed."""
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        name = re.compile(r"void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\([^{};]*\)\s*\{").search(text, m.end())
        depth, at = 1, name.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield name.group(1), text[name.end():at - 1]


def cluster_kernels():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                out += [(f, n, b) for n, b in kernels(fh.read()) if "map_shared_rank" in b]
    return out


def test_kernels_are_found():
    assert {"k_sqminl_panel", "k_sqminl_panel_sm"} <= {n for _, n, _ in cluster_kernels()}


@pytest.mark.parametrize("f,name,body", cluster_kernels(), ids=lambda v: v if "\n" not in v else "body")
def test_barrier_before_first_mapping(f, name, body):
    mapped = body.index("map_shared_rank")
    store = re.search(r"\*\s*cl\.map_shared_rank\([^;]*\)\s*=(?!=)", body)
    barrier = re.search(r"\bcl\.sync\(\)", body)
    assert barrier and barrier.start() < mapped, name
    if store:   # a pushing kernel: its peers are waited for before the loop of exchanges
        before = body[:barrier.start()]
        assert before.count("{") == before.count("}"), name
