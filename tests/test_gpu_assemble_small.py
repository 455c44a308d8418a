"""Direct assembly of operators that take 64-thread CTAs (fewer than 152 CTAs of
256 threads) and of the first ones that do not: the mixed form's two words against the FP64
values, full and reduced, and the reduced CFIE against the full operator folded
over its orbits, at real and complex wavenumbers. Every kernel computes the
same FP64 entries up to rounding, hi + lo carries 2^-48 of each, and an orbit has
four: within 1e-13 of the max-norm, as the other assembly tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = [20, 62, 190, 192, 194, 258]


def _both(qb, ws, ks):
    ref = qb.assemble(ws, ks)
    out = qb.assemble(ws, ks, mixed=True, split_lo=True)
    for q in range(len(ks)):
        v = out[q].astype(np.complex128) + out[len(ks) + q].astype(np.complex128)
        assert np.abs(v - ref[q]).max() <= 1e-13 * np.abs(ref[q]).max(), q
    return ref


@pytest.mark.parametrize("n", N)
@pytest.mark.parametrize("form", ["dlp", "cfie"])
def test_full(qb, n, form):
    b = qb.make_circle(1.0) if form == "dlp" else qb.make_star(0.2, 5)
    pts, sol = qb.points_with_n((qb.DLP_kress if form == "dlp" else qb.CFIE_kress)(1.0, b), b, n, 0.08 * n)
    _both(qb, qb.Workspace(sol, pts), [0.08 * n, 0.08 * n + 0.3j, 0.08 * n + 2j])


@pytest.mark.parametrize("m", N)
@pytest.mark.parametrize("form", ["dlp", "cfie"])
def test_reduced(qb, m, form):
    b = qb.make_full_stadium(1.0, 1.0)
    make = qb.DLP_kress_global_corners if form == "dlp" else qb.CFIE_kress_global_corners
    k = 0.08 * m
    pts, sol = qb.points_with_n(make(1.0, b, symmetry=qb.XYReflection(1, -1)), b, 4 * m, k)
    ws = qb.Workspace(sol, pts)
    assert ws.dim == m
    ref = _both(qb, ws, [k, k + 0.3j, k + 2j])
    if form == "cfie":
        fund, orbit, scale = ws._red[0], ws._red[1], ws._red[2].view(np.complex128).reshape(ws._red[1].shape)
        full, solf = qb.points_with_n(make(1.0, b), b, 4 * m, k)
        A = qb.assemble(qb.Workspace(solf, full), [k, k + 0.3j, k + 2j])
        for q in range(3):
            fold = np.zeros((m, m), complex)
            for c in range(m):
                for l in range(orbit.shape[1]):
                    fold[:, c] += scale[c, l] * A[q][fund, orbit[c, l]]
            assert np.abs(fold - ref[q]).max() <= 1e-13 * np.abs(ref[q]).max(), q
