"""Jobs whose faster solve the server's memory budget does not hold run in the
smaller form instead of being refused: the footprint is the smaller one and the
parameters are those of the job in the faster form, within the 1e-9 of
test_gpu_bspmv (condition below 1e4, residual test at 1e-13)."""
import numpy as np
import pytest
from test_gpu_bspmv import SIZES, records

pytestmark = pytest.mark.gpu


def run(mp, d, budget, **st):
    jd = mp.JobData(d, mitera=1, mreqenf=1, mreqena=1, mrestl=1e-13, **st)
    with mp.Server(max_active=1, budget_bytes=budget) as srv:
        rc, _, _, b = srv.wait(srv.submit(jd), timeout_ms=600000.0)
    return rc, b, jd


@pytest.mark.parametrize("name", ["1", "3", "6", "5-6"])
@pytest.mark.parametrize("metsol", [4, 5])
def test_sparse_product_without_the_copy(mp, name, metsol):
    d, n = records(SIZES[name], 170, 700, 11)
    labels = np.arange(1, n + 1, dtype=np.int32)
    st = dict(params=(labels, np.zeros(n), np.full(n, 5.0 ** -0.5)), metsol=metsol, matsto=2)
    rc, full, jd = run(mp, d, 0, **st)
    assert rc == 0
    _, want = jd.parameters()
    assert np.max(np.abs(want)) > 0
    rc, b, jd = run(mp, d, full - 1, **st)
    assert rc == 0 and b < full
    _, got = jd.parameters()
    assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))
    rc, _, _ = run(mp, d, b - 1, **st)
    assert rc == 42


def test_slices_of_the_inverse(mp):
    """The blocked FP64 inversion: the footprint holds the slices of both
    operands (24 bytes per element, all K tiles below 64); in windows of four
    K tiles where the budget does not, with the same solution."""
    cfg = mp.gen_config("telescope", ntracks=20000, seed=22)
    cfg.nmod = 80
    d = mp.generate(cfg)
    st = dict(metsol=12, matsto=1)
    rc, full, jd = run(mp, d, 0, **st)
    assert rc == 0
    labels, want = jd.parameters()
    npad = (len(labels) + 127) // 128 * 128
    assert npad > 5 * 128
    rc, b, jd = run(mp, d, full - 1, **st)
    assert rc == 0 and full - b >= 2 * 24 * npad * npad
    np.testing.assert_array_equal(jd.parameters()[1], want)   # the solution does not take the inverse
    rc, _, _ = run(mp, d, b - 1, **st)
    assert rc == 42
