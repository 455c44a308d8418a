"""The 32-column FP64 panels of the library's own operators, on clusters of 4 and
8 CTAs (as many as the batch leaves SMs for; other sizes in test_gpu_sigma_lu) and
with 1, 2 and 33 columns left for the last panel: sigma_min of every operator
against LAPACK, which a backward-stable factorisation meets to a few eps
sigma_max. Matrices that a caller hands in take 64-column panels: the same
operators inverted through that entry, against the identity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [34, 66, 98, 130, 290])
@pytest.mark.parametrize("nk", [19, 38])
def test_both_panel_widths(qb, n, nk):
    from qbgpu import _lib as L
    c = qb.make_star(0.2, 5)
    k = 0.08 * n
    pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, n, k)
    ws = qb.Workspace(sol, pts)
    ks = k + 0.02 * np.arange(nk)
    sig = qb.sigma_min(ws, ks)
    A = np.array([qb.assemble(ws, [x])[0] for x in ks])
    s = np.linalg.svd(A, compute_uv=False)
    assert np.max(np.abs(sig - s[:, -1]) / s[:, 0]) <= 2e-14
    a = np.ascontiguousarray(A.transpose(0, 2, 1))
    x = np.empty_like(a)
    m = a.shape[1]
    L.check(L.load().qbg_dense_inverse(m, nk, L.QBG_PREC_FP64, L.vptr(a), L.vptr(x), None, None))
    X = x.transpose(0, 2, 1)
    eye = np.eye(m)
    for q in range(nk):
        assert np.linalg.norm(A[q] @ X[q] - eye, 2) <= 16 * m * 2.0 ** -52 * s[q, 0] / s[q, -1], q
