"""The blocked FP64 inversion (metsol 12 with errors) at sizes around its tiles
of 128 and scale groups of 512 against numpy's inverse.  Eigenvalues between 1
and 7: solution and diagonal within 10 n cond(A) u of the largest element."""
import numpy as np
import pytest
from test_gpu_packed import context, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 127, 130, 384, 511, 520, 650, 1100])
def test_blocked_inverse(mp, n):
    M, b = matrix(n, n, 0)
    with context(mp, n, M, b) as ctx:
        p = ctx.matrix()
        g = np.zeros(n)
        ctx.check(ctx.L.mpgpu_download_vector(ctx.h, mp.ptr(g, mp.f64p), None))
        x, err, info = ctx.solve(12, errors=True)
    A = np.zeros((n, n))
    A[np.tril_indices(n)] = p
    A = A + np.tril(A, -1).T
    inv = np.linalg.inv(A)
    tol = 10 * n * 7 * 2.0 ** -53
    assert info.nrank == n
    assert np.max(np.abs(x - inv @ g)) <= tol * np.max(np.abs(inv @ g))
    assert np.max(np.abs(err - np.diag(inv))) <= tol * np.max(np.diag(inv))
