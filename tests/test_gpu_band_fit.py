"""Band records of the data loop around the limits of their forms: the Schur
term from the factors (up to 8 border locals and 4 bands; the full inverse
beyond), batched normal equations (up to 10 locals per equation), equations
with globals in ones, whole and partial warps, groups of several sizes, both
border sides, small and large-record kernels; against the oracle, decisions
exactly and sums within 1e-12 as in test_gpu_loopbf."""
import numpy as np
import pytest

from test_gpu_loopbf import check

pytestmark = pytest.mark.gpu


def records(border, width, nloc, ngeq, side, sizes, seed, nrec=60, repeat=False):
    """nrec records of nloc locals: every equation holds the border locals
    (the first ones, or the last for side 2) and width + 1 consecutive band
    locals; ngeq equations with globals, two per crossed group (`repeat`:
    groups crossed again), then equations without globals."""
    rng = np.random.default_rng(seed)
    ngroups = 40
    size = [sizes[g % len(sizes)] for g in range(ngroups)]
    first = np.concatenate([[0], np.cumsum(size)])
    ptr, ind, val = [0], [], []
    nband = nloc - border
    for _ in range(nrec):
        ind.append(0)
        val.append(0.0)
        order = rng.permutation(ngroups)
        neq = max(ngeq, 0) + nloc + 6
        for e in range(neq):
            s = int(e * (nband - width - 1) / max(neq - 1, 1)) if nband > width + 1 else 0
            band = np.arange(s, min(s + width + 1, nband)) + 1
            loc = np.concatenate([np.arange(1, border + 1), band + border]) if side == 1 else \
                np.concatenate([band, np.arange(nband + 1, nloc + 1)])
            ind += [0] + loc.tolist() + [0]
            val += [rng.normal()] + (rng.normal(size=len(loc)) + 0.5).tolist() + [0.3 + rng.random()]
            if e < ngeq:
                g = order[(e // 2) % (7 if repeat else ngroups)]
                ind += list(range(first[g] + 1, first[g + 1] + 1))
                val += rng.normal(size=size[g]).tolist()
        ptr.append(len(ind))
    return dict(recPtr=np.array(ptr, np.int64), inder=np.array(ind, np.int32), glder=np.array(val))


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("border,width,nloc,ngeq,side,sizes,repeat", [
    (4, 3, 12, 2, 1, [6], False), (4, 3, 40, 31, 1, [6], False), (4, 3, 40, 32, 1, [6], False),
    (4, 3, 40, 33, 1, [6], False), (4, 3, 64, 64, 1, [6, 5], False), (4, 2, 84, 66, 1, [6], True),
    (0, 2, 20, 20, 1, [3], False), (0, 4, 20, 20, 1, [1, 2], False), (8, 1, 30, 24, 1, [6], False),
    (8, 4, 40, 24, 1, [6], False), (9, 1, 30, 24, 1, [6], False), (4, 5, 40, 24, 1, [6], False),
    (1, 9, 40, 24, 1, [6], False), (3, 2, 30, 33, 2, [6], False), (3, 3, 40, 40, 2, [4, 8], True)])
def test_band_records(mp, orc, flags, border, width, nloc, ngeq, side, sizes, repeat):
    d = records(border, width, nloc, ngeq, side, sizes, border + 10 * width + nloc, repeat=repeat)
    for opt in (dict(), dict(nloopn=2, lhuber=3)):
        H = mp.HostStructure(d, mreqenf=1, sparse=True)
        O = orc.Structure(d, mreqenf=1, sparse=True)
        gpar = np.zeros(H.nTotal)
        o = O.loopbf(gpar, matsto=2, **opt)
        with mp.Context(flags=flags) as ctx:
            ctx.set_layout(H, 2)
            ctx.upload(H)
            g = ctx.loopbf(gpar, **opt)
            g["matD"] = ctx.matrix()
            g["status"] = ctx.status()
        assert np.sum(o["status"] == 0) > 30
        check(g, o)
