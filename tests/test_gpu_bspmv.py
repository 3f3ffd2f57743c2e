"""Sparse product and MINRES on layouts with parameter groups of every size
the block-row copy takes (1 to 8), mixed sizes with little padding, sizes it
leaves to the other kernels (strongly mixed, above 8), and with numbers of
constraints around the limit of the fused reflections: against the same
matrix in packed storage, dense on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {"1": [1], "2": [2], "3": [3], "4": [4], "5": [5], "6": [6], "7": [7], "8": [8], "5-6": [5, 6, 6],
         "1-8": [1, 1, 1, 8], "9": [9, 3]}


def records(sizes, ngroups, ntracks, seed):
    """Tracks crossing 2 to 7 of the groups, two locals, two measurements per
    crossing with random derivatives of every parameter of the group; a
    hub group crossed by every second track (long rows)."""
    rng = np.random.default_rng(seed)
    size = [sizes[g % len(sizes)] for g in range(ngroups)]
    first = np.concatenate([[0], np.cumsum(size)])
    ptr, ind, val = [0], [], []
    for t in range(ntracks):
        hit = set(rng.integers(0, ngroups, rng.integers(2, 8)).tolist()) | ({0} if t % 2 else set())
        ind.append(0)
        val.append(0.0)
        for g in sorted(hit):
            for _ in range(2):
                ind += [0, 1, 2, 0] + list(range(first[g] + 1, first[g + 1] + 1))
                val += [rng.normal(), rng.normal(), rng.normal(), 0.5] + rng.normal(size=size[g]).tolist()
        ptr.append(len(ind))
    return dict(recPtr=np.array(ptr, np.int64), inder=np.array(ind, np.int32), glder=np.array(val)), int(first[-1])


def dense(ctx, n):
    M = np.zeros((n, n))
    M[np.tril_indices(n)] = ctx.matrix()
    return M + np.tril(M, -1).T


def build(mp, d, matsto, A):
    H = mp.HostStructure(d, mreqenf=1, sparse=matsto == 2)
    ctx = mp.Context()
    ctx.set_layout(H, matsto)
    if A is not None:
        ctx.set_constraints(A)
    ctx.upload(H)
    lb = ctx.loopbf(np.zeros(H.nTotal))
    iv = np.arange(1, H.nVar + 1, dtype=np.int32)
    ctx.mupdat(iv, iv, np.full(H.nVar, 5.0))
    return ctx, lb["gvec"]


@pytest.mark.parametrize("name", list(SIZES))
@pytest.mark.parametrize("ngroups,ntracks", [(3, 40), (40, 400), (170, 700)])
def test_product(mp, name, ngroups, ntracks):
    """avprod without constraints: two summation orders of at most 2 n terms,
    so 1e-13 of the absolute row products."""
    d, n = records(SIZES[name], ngroups, ntracks, 7)
    x = np.random.default_rng(1).normal(size=n)
    with build(mp, d, 1, None)[0] as ctx:
        M = dense(ctx, n)
    with build(mp, d, 2, None)[0] as ctx:
        b = ctx.avprod(x)
    assert np.all(np.abs(b - M @ x) <= 1e-13 * (np.abs(M) @ np.abs(x)))


@pytest.mark.parametrize("name", ["1", "3", "6", "5-6", "1-8", "9"])
@pytest.mark.parametrize("ncon", [0, 1, 18, 64, 65])
@pytest.mark.parametrize("metsol,mbandw", [(4, 0), (5, 0), (4, 3), (4, -1)])
def test_minres(mp, name, ncon, metsol, mbandw):
    """Solutions against the KKT system of the dense matrix; condition below
    1e4 after the added diagonal, residual test at 1e-13: 1e-9 relative."""
    d, n = records(SIZES[name], 170, 700, 11)
    A = np.random.default_rng(2).normal(size=(ncon, n)) if ncon else None
    with build(mp, d, 1, None)[0] as ctx:
        M = dense(ctx, n)
    ctx, g = build(mp, d, 2, A)
    rhs = np.random.default_rng(3).normal(size=ncon)
    with ctx:
        ctx.set_preconditioner(mbandw)
        x, _, info = ctx.solve(metsol, consResiduals=rhs if ncon else None, rtol=1e-13, itnlim=3000)
    K = np.block([[M, A.T], [A, np.zeros((ncon, ncon))]]) if ncon else M
    want = np.linalg.solve(K, np.concatenate([g, rhs]))[:n]
    assert info.istop in (1, 2)
    assert np.max(np.abs(x - want)) <= 1e-9 * np.max(np.abs(want))
