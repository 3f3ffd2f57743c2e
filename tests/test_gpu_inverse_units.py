"""The blocked FP64 inversion (metsol 12 with errors) of a matrix whose
parameters have different units: A = D A' D with D powers of two, so that every
step of an FP64 factorisation and inversion scales exactly and the relative
errors are those of A' (eigenvalues between 1 and 7: 10 n cond(A') u of the
largest element), element by element whatever D.  Sizes below one super-block
(512 rows), with one, two and three doublings above it."""
import numpy as np
import pytest
from test_gpu_packed import context, matrix

pytestmark = pytest.mark.gpu


def exponents(n, units):
    if units.startswith("group"):   # three of six parameters per module
        return int(units[5:]) * (np.arange(n) % 6 < 3)
    return np.random.default_rng(n).integers(0, int(units[6:]), n)


@pytest.mark.parametrize("units", ["group7", "group20", "group27", "random50", "random100"])
@pytest.mark.parametrize("n", [130, 300, 650, 1100, 2100])
def test_errors_do_not_depend_on_units(mp, n, units):
    s = np.ldexp(1.0, exponents(n, units))
    M, b = matrix(n, n, 0)
    with context(mp, n, M * s[:, None] * s[None, :], b * s) as ctx:
        p = ctx.matrix()
        _, err, info = ctx.solve(12, errors=True)
    A = np.zeros((n, n))
    A[np.tril_indices(n)] = p
    A = (A + np.tril(A, -1).T) / s[:, None] / s[None, :]
    diag = np.diag(np.linalg.inv(A))
    tol = 10 * n * 7 * 2.0 ** -53
    assert info.nrank == n
    assert np.max(np.abs(err * s * s - diag)) <= tol * np.max(diag)
