"""Direct FP64 assembly by node pairs against the oracle: sizes below and above
the change from single entries to pairs, off the 16-node tiles, one wavenumber
and several (which the launch spreads over the grid), real and complex
ones, A alone and with its derivatives, one component and two. The
bound is that of the other FP64 assembly tests, 1e-12 of the max-norm."""
import numpy as np
import pytest

from oracle import assembly as OA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(20, 1), (30, 9), (128, 1), (130, 3), (242, 1), (258, 2), (300, 1), (64, 70)])
@pytest.mark.parametrize("form", ["dlp", "cfie"])
@pytest.mark.parametrize("deriv", [False, True])
def test_direct_assembly(qb, n, nk, form, deriv):
    b = qb.make_star() if form == "dlp" else qb.make_circle_with_hole()
    sol = (qb.DLP_kress if form == "dlp" else qb.CFIE_kress)(1.0, b)
    pts, sol = qb.points_with_n(sol, b, n, 0.1 * n)
    ws = qb.Workspace(sol, pts)
    k = max(2.0, 0.1 * n)
    for ks in (k + 0.01 * np.arange(nk), k + 0.01 * np.arange(nk) + 0.3j):
        got = qb.assemble(ws, ks, deriv=deriv)
        for q in sorted({0, nk - 1}):
            ref = OA.assemble(form, pts, ks[q] if np.iscomplexobj(ks) else float(ks[q]), derivs=deriv)
            ref = ref if deriv else (ref,)
            for v, r in enumerate(ref):
                assert np.abs(got[v * nk + q] - r).max() <= 1e-12 * np.abs(r).max(), (q, v)
