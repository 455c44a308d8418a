"""sigma_min of a sweep (Lanczos on the LU factors, one cluster of CTAs per
operator) against LAPACK singular values of the same matrices, at the edges of
its 64-row blocks and of the cluster sizes: one operator up to eight CTAs, a
batch that takes one CTA each, operators of a single block. A backward-stable
sigma_min is exact to a few eps sigma_max in absolute terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(20, 1), (20, 70), (62, 3), (64, 40), (66, 2), (128, 160), (130, 80), (194, 310), (258, 5), (514, 1), (578, 2)])
@pytest.mark.parametrize("form", ["dlp", "cfie"])
def test_sigma_min_matches_lapack(qb, form, n, nk):
    b = qb.make_circle(1.0) if form == "dlp" else qb.make_star()
    sol = (qb.DLP_kress if form == "dlp" else qb.CFIE_kress)(1.0, b)
    k = 0.08 * n
    pts, sol = qb.points_with_n(sol, b, n, k)
    ws = qb.Workspace(sol, pts)
    ks = np.linspace(k, k + 0.7, nk) if nk > 1 else np.array([k])
    sig = qb.sigma_min(ws, ks)
    for q in sorted({0, nk // 2, nk - 1}):
        s = np.linalg.svd(qb.assemble(ws, [ks[q]])[0], compute_uv=False)
        assert abs(sig[q] - s[-1]) <= 2e-14 * s[0], (q, sig[q], s[-1])
