"""J/E tables of the mixed-form assembly at the edges of their build: one to a few
panels (all sampled at the Lobatto points), panel counts at and off the 32 of a
CTA, panels wide enough (|k h| > 1.5) to be sampled, the highest degree, real and
complex wavenumbers. hi + lo against the FP64 direct assembly; degree 16 resolves
|k h| <= 1.8 to 1e-15, so the bound is that of the other double-float assembly
tests, 1e-13 of the max-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["dlp", "cfie"])
@pytest.mark.parametrize("k,n_j", [(2.0, 1), (3.0, 2), (6.0, 3), (20.0, 9), (20.0, 21), (20.0, 22), (20.0, 43), (60.0, 400)])
@pytest.mark.parametrize("im", [0.0, 0.3])
def test_je_tables(qb, form, k, n_j, im):
    b = qb.make_star(0.2, 5)
    sol = (qb.DLP_kress if form == "dlp" else qb.CFIE_kress)(1.0, b)
    pts, sol = qb.points_with_n(sol, b, 200, k)
    ws = qb.Workspace(sol, pts)
    ks = [k + 1j * im, k - 0.1 - 1j * im]
    ref = qb.assemble(ws, ks)
    out = qb.assemble(ws, ks, mixed=True, cheb=(500, 9, n_j, 16), split_lo=True)
    for q in range(2):
        v = out[q].astype(np.complex128) + out[2 + q].astype(np.complex128)
        assert np.abs(v - ref[q]).max() <= 1e-13 * np.abs(ref[q]).max(), q
