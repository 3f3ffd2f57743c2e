"""Warps per CTA of a class that is not sampled: the same in the first loop of
a process as in later ones, at record sizes where CTAs of several warps (more
shared memory than a kernel has without opting in) hold more warps per SM."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
import numpy as np
sys.path.insert(0, {tests!r})
from conftest import load_pkg_module
mp = load_pkg_module("mpgpu")
hits, per = {hits}, {per}
rng = np.random.default_rng(1)
ptr, ind, val = [0], [], []
for t in range(200):
    ind.append(0)
    val.append(0.0)
    for g in sorted(rng.choice(60, hits, False).tolist()):
        for _ in range(per):
            ind += [0, 1, 2, 0] + list(range(6 * g + 1, 6 * g + 7))
            val += [rng.normal()] + rng.normal(size=2).tolist() + [0.5] + rng.normal(size=6).tolist()
    ptr.append(len(ind))
d = dict(recPtr=np.array(ptr, np.int64), inder=np.array(ind, np.int32), glder=np.array(val))
S = mp.HostStructure(d, mreqenf=1, sparse=True)
for _ in range(2):
    with mp.Context() as ctx:
        ctx.set_layout(S, 2)
        ctx.upload(S)
        ctx.loopbf(np.zeros(S.nTotal))
        print(ctx.fit_buckets()[1].tolist())
"""


@pytest.mark.parametrize("hits,per", [(20, 2), (27, 2), (30, 1)])
def test_first_loop_takes_the_form_of_later_ones(mp, hits, per):
    tests = os.path.dirname(os.path.abspath(__file__))
    out = subprocess.run([sys.executable, "-c", PROGRAM.format(tests=tests, hits=hits, per=per)], check=True,
                         capture_output=True, text=True, timeout=300).stdout.split("\n")
    assert out[0] == out[1]
    assert max(eval(out[0])) > 1   # a size where it matters
