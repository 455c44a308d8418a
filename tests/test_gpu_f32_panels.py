"""complex64 LU on the cluster panels: every cluster size (1 to 16 CTAs), row
counts at and around the rows a CTA holds, sub-panels and panels that end
early, one operator and several. The cluster panels pivot exactly as the
one-CTA ones, so the explicit inverses agree to FP32 rounding; both against the
identity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inverse(qb, A, cluster):
    from qbgpu import _lib as L
    lib = L.load()
    o, c, p = (L.C.c_int32() for _ in range(3))
    L.check(lib.qbg_get_lu_plan(L.C.byref(o), L.C.byref(c), L.C.byref(p)))
    batch, n, _ = A.shape
    a = np.ascontiguousarray(A.transpose(0, 2, 1))
    x = np.empty_like(a)
    try:
        L.check(lib.qbg_set_lu_plan(0, cluster, 0))
        L.check(lib.qbg_dense_inverse(n, batch, L.QBG_PREC_FP32, L.vptr(a), L.vptr(x), None, None))
    finally:
        L.check(lib.qbg_set_lu_plan(0, c.value, 0))
    return x.transpose(0, 2, 1)


@pytest.mark.parametrize("n,batch", [(1, 2), (8, 1), (64, 2), (65, 3), (71, 1), (255, 2), (257, 1), (399, 2), (400, 1), (401, 2),
                                     (799, 1), (801, 1), (1599, 1), (1603, 1), (3201, 1)])
def test_inverse_matches_the_one_cta_panels(qb, n, batch):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))) / np.sqrt(n)
    A += 2.5 * np.eye(n)[rng.permutation(n)]  # every column pivots
    X = _inverse(qb, A, 1)
    for b in range(batch):
        assert np.abs(A[b] @ X[b] - np.eye(n)).max() < 2e-5, b
    assert np.abs(X - _inverse(qb, A, 0)).max() < 2e-5


def test_ties_zero_columns_and_nan(qb):
    n = 130
    A = np.zeros((2, n, n), complex)
    A[0] = np.fliplr(np.eye(n))  # one exact pivot per column, in the last row left
    A[1] = np.eye(n) + np.tri(n, k=-1)  # equal magnitudes: the first index wins
    for c in (0, 1):
        X = _inverse(qb, A, c)
        for b in range(2):
            assert np.abs(A[b] @ X[b] - np.eye(n)).max() < 1e-5
    A[0, 3, 5] = np.nan
    X = _inverse(qb, A, 1)
    assert np.isnan(X[0]).any() and np.abs(A[1] @ X[1] - np.eye(n)).max() < 1e-5
