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


@pytest.mark.parametrize("n", [8300, 16600])   # X^T X; the block inverses too
def test_inverse_in_windows(mp, n):
    """More K tiles than the sliced operands hold at a time: a diagonal plus
    eight dyads, whose inverse is known (eigenvalues between 1 and 8)."""
    rng = np.random.default_rng(5)
    d = rng.uniform(1.0, 3.0, n)
    V = 2.0 * rng.normal(size=(n, 8)) / np.sqrt(n)
    M = V @ V.T
    M[np.arange(n), np.arange(n)] += d
    with context(mp, n, M, rng.normal(size=n)) as ctx:
        g = np.zeros(n)
        ctx.check(ctx.L.mpgpu_download_vector(ctx.h, mp.ptr(g, mp.f64p), None))
        x, err, info = ctx.solve(12, errors=True)
    W = V / d[:, None]
    C = np.linalg.inv(np.eye(8) + V.T @ W)
    xr, diag = g / d - W @ (C @ (W.T @ g)), 1.0 / d - np.einsum("ik,kl,il->i", W, C, W)
    tol = 10 * n * 8 * 2.0 ** -53
    assert info.nrank == n
    assert np.max(np.abs(x - xr)) <= tol * np.max(np.abs(xr))
    assert np.max(np.abs(err - diag)) <= tol * np.max(diag)
