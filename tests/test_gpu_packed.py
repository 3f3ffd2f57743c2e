"""pede's inversion and decomposition of the packed matrix (metsol 1 and 3) at
sizes around their blocks of pivots, update tiles and cluster sizes, against
the oracle's sqminl and chdec2/chslv2 of the same matrix: rank equal, solution
and errors within 1e-10 of a well-conditioned matrix (the same operations per
element up to fused products)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(mp, n, M, b):
    """Context whose matrix is M and vector b: a layout of n labels, one loop
    of a record per label, then the differences added."""
    ptr, ind, val = [0], [], []
    for lab in range(1, n + 1):
        ind += [0, 0, 1, 0, lab, 0, 1, 0, lab]
        val += [0.0, 0.1, 1.0, 1.0, 1.0, -0.1, 1.0, 1.0, 2.0]
        ptr.append(len(ind))
    d = dict(recPtr=np.array(ptr, np.int64), inder=np.array(ind, np.int32), glder=np.array(val))
    H = mp.HostStructure(d, mreqenf=1, sparse=False)
    assert H.nVar == n
    ctx = mp.Context()
    ctx.set_layout(H, 1)
    ctx.upload(H)
    lb = ctx.loopbf(np.zeros(n))
    i, j = np.tril_indices(n)
    ctx.mupdat(i + 1, j + 1, M[i, j] - ctx.matrix())
    iv = np.arange(1, n + 1, dtype=np.int32)
    add = b - lb["gvec"]
    ctx.check(ctx.L.mpgpu_vector_add(ctx.h, C.c_int32(n), mp.ptr(iv, mp.i32p), mp.ptr(add, mp.f64p)))
    return ctx


def matrix(n, seed, deficient):
    rng = np.random.default_rng(seed)
    B = rng.normal(size=(n, n + 5))
    M = B @ B.T / n + np.diag(rng.uniform(1.0, 3.0, n))
    for k in range(deficient):   # zero rows: no pivot for them
        M[3 * k + 1, :] = 0.0
        M[:, 3 * k + 1] = 0.0
    return M, rng.normal(size=n)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 130, 512, 513, 1025, 1100])
@pytest.mark.parametrize("metsol,deficient", [(1, 0), (3, 0), (1, 3)])
def test_packed(mp, orc, n, metsol, deficient):
    if deficient and n < 3 * deficient:
        pytest.skip("fewer rows than dependent ones")
    M, b = matrix(n, n, deficient)
    with context(mp, n, M, b) as ctx:
        A = ctx.matrix()
        g = np.zeros(n)
        ctx.check(ctx.L.mpgpu_download_vector(ctx.h, mp.ptr(g, mp.f64p), None))
        x, err, info = ctx.solve(metsol, errors=metsol == 1)
    L, xo, nr = orc.lib(), g.copy(), C.c_int32()
    if metsol == 1:
        L.mpref_sqminl(orc.ptr(A, orc.f64p), orc.ptr(xo, orc.f64p), C.c_int32(n), C.byref(nr))
    else:
        emax, emin = C.c_double(), C.c_double()
        L.mpref_chdec2(orc.ptr(A, orc.f64p), C.c_int32(n), C.byref(nr), C.byref(emax), C.byref(emin))
        L.mpref_chslv2(orc.ptr(A, orc.f64p), orc.ptr(xo, orc.f64p), C.c_int32(n))
        assert abs(info.evmax - emax.value) <= 1e-12 * emax.value
        assert abs(info.evmin - emin.value) <= 1e-12 * emin.value
    assert info.nrank == nr.value == n - deficient
    assert np.max(np.abs(x - xo)) <= 1e-10 * np.max(np.abs(xo))
    if metsol == 1:
        diag = A[np.cumsum(np.arange(1, n + 1)) - 1]
        assert np.max(np.abs(err - diag)) <= 1e-10 * np.max(np.abs(diag))


def test_inversion_above_one_row_per_thread(mp):
    """More rows than the threads of the largest cluster, against numpy:
    eigenvalues between 1 and 7, within 10 n cond(A) u."""
    n = 4200
    M, b = matrix(n, 4, 0)
    with context(mp, n, M, b) as ctx:
        p = ctx.matrix()
        g = np.zeros(n)
        ctx.check(ctx.L.mpgpu_download_vector(ctx.h, mp.ptr(g, mp.f64p), None))
        x, err, info = ctx.solve(1, errors=True)
    A = np.zeros((n, n))
    A[np.tril_indices(n)] = p
    A = A + np.tril(A, -1).T
    inv = np.linalg.inv(A)
    tol = 10 * n * 7 * 2.0 ** -53
    assert info.nrank == n
    assert np.max(np.abs(x - inv @ g)) <= tol * np.max(np.abs(inv @ g))
    assert np.max(np.abs(err - np.diag(inv))) <= tol * np.max(np.diag(inv))
