"""The FP64 dense Cholesky (mpgpu_dense_cholesky, mode 0) at sizes around its
launches of 32 columns, panels of 128 and block columns of 512, on dense,
spiky and badly scaled matrices: |A - L L^T| within 3 (n + 2) u of
sqrt(a_ii a_jj), the bound of a Cholesky factorisation in floating point
(gamma_(n+1) |L| |L|^T, and |L| |L|^T is below sqrt(a_ii a_jj); u = 2^-53) with
3 in place of 1 for the reciprocals and roots in the products.  Pivots beyond
the range of the fast root, and matrices that are not positive definite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(n, kind):
    rng = np.random.default_rng(n)
    if kind == "dense":
        B = rng.normal(size=(n, n + 10))
        return B @ B.T / n
    if kind == "scaled":
        s = 2.0 ** rng.integers(-50, 50, n)
        return matrix(n, "dense") * s[:, None] * s[None, :]
    M = np.zeros((n, n))   # a few large elements per row, as records give them
    for _ in range(4 * n):
        i = rng.choice(n, min(n, 12), False)
        g = rng.normal(size=len(i)) * 10.0 ** rng.uniform(-2, 2, len(i))
        M[np.ix_(i, i)] += np.outer(g, g)
    return M + np.diag(1e-3 * np.diag(M) + 1e-6)


# (2,700 and 5,400 rows: the first panels take four lanes per row, the last eight)
@pytest.mark.parametrize("n,kind", [(n, kind) for kind in ("dense", "scaled", "spiky")
                                    for n in (1, 31, 33, 96, 127, 129, 160, 385, 513, 650, 1160)]
                         + [(2700, "scaled"), (5400, "dense")])
def test_backward_error(mp, n, kind):
    A = matrix(n, kind)
    with mp.Context() as ctx:
        L, _ = ctx.dense_cholesky(A, 0)
    rows = np.unique(np.linspace(0, n - 1, 60).astype(int))
    Lx = L.astype(np.longdouble)
    d = np.sqrt(np.diag(A))
    err = np.abs(A[rows] - Lx[rows] @ Lx.T) / (d[rows][:, None] * d[None, :])
    assert np.max(err) <= 3 * (n + 2) * 2.0 ** -53


@pytest.mark.parametrize("scale", [2.0 ** -600, 2.0 ** -130, 2.0 ** 130, 2.0 ** 900])
def test_pivot_range(mp, scale):
    """Scaling by a power of 4 scales every operation exactly."""
    n = 200
    A = matrix(n, "dense")
    with mp.Context() as ctx:
        L, _ = ctx.dense_cholesky(A * scale, 0)
    d = np.sqrt(np.diag(A))
    L = L / np.sqrt(scale)
    assert np.max(np.abs(A - L @ L.T) / (d[:, None] * d[None, :])) <= 6 * (n + 2) * 2.0 ** -53


@pytest.mark.parametrize("row", [0, 31, 32, 100, 128, 700])
def test_not_positive_definite(mp, row):
    A = matrix(780, "dense")
    A[row, row] = -1.0
    with mp.Context() as ctx:
        for mode in (0, 1):
            with pytest.raises(RuntimeError, match="non-positive pivot"):
                ctx.dense_cholesky(A, mode)
        L, _ = ctx.dense_cholesky(matrix(130, "dense"), 0)   # the context works on
    assert np.all(np.isfinite(L))
