"""Ordered additions of mpgpu_mupdat and mpgpu_vector_add at the sizes where
their chunks and rounds end: no term is lost, and the terms of one element
are added in the order of the call, bit for bit as one thread adds them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 4095, 4096, 4097, 9001])
@pytest.mark.parametrize("spread", [1, 3, 40, 20100])
def test_order_of_terms(mp, n, spread):
    """n terms on `spread` packed elements (1: all on one, the sequential end
    of a chunk) and as many on the vector; the sums depend on the order
    (terms of 1e-8 to 1e8), so equality is exact."""
    d = mp.generate(mp.gen_config("telescope", ntracks=200, seed=3))
    H = mp.HostStructure(d, mreqenf=1, sparse=False)
    rng = np.random.default_rng(n + spread)
    i, j = np.tril_indices(H.nVar)
    pick = rng.integers(0, min(spread, len(i)), n)
    add = rng.normal(size=n) * 10.0 ** rng.integers(-8, 9, n)
    iv, jv = (i[pick] + 1).astype(np.int32), (j[pick] + 1).astype(np.int32)
    with mp.Context() as ctx:
        ctx.set_layout(H, 1)
        ctx.upload(H)
        lb = ctx.loopbf(np.zeros(H.nTotal))
        want, vwant = ctx.matrix(), lb["gvec"].copy()
        ctx.mupdat(jv, iv, add)   # either order of the two indices
        ctx.check(ctx.L.mpgpu_vector_add(ctx.h, mp.C.c_int32(n), mp.ptr(iv, mp.i32p), mp.ptr(add, mp.f64p)))
        got = ctx.matrix()
        vgot = np.zeros(H.nVar)
        ctx.check(ctx.L.mpgpu_download_vector(ctx.h, mp.ptr(vgot, mp.f64p), None))
    for q in range(n):
        want[pick[q]] += add[q]
        vwant[iv[q] - 1] += add[q]
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(vgot, vwant)
