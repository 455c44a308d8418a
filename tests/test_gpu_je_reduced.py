"""Mixed-form assembly of the reduced DLP, double-float words hi + lo against
the FP64 direct assembly: orbits of two and four nodes (on the J/E tables) and
of three and five, or with complex scales, or panels of degree 5 (on the H and J
tables), reduced orders below, at and off the 32 x 16 entry tiles, one
wavenumber and several. The panels resolve both interpolants beyond 1e-14, so
the bound is that of the other double-float assembly tests, 1e-13 of the
max-norm; with degree 5 it is held against the FP64 assembly of the same panels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sym(qb, name):
    kind, *a = name
    return {"x": qb.XReflection, "xy": qb.XYReflection, "rot": qb.Rotation}[kind](*a)


@pytest.mark.parametrize("sym", [("x", 1), ("x", -1), ("xy", -1, 1), ("xy", 1, 1), ("rot", 2, 1), ("rot", 4, 0),
                                 ("rot", 3, 1), ("rot", 5, 0)])
@pytest.mark.parametrize("n", [40, 128, 500])
@pytest.mark.parametrize("deg", [5, 7, 9])
def test_reduced_mixed_assembly(qb, sym, n, deg):
    rot = sym[0] == "rot"
    b = qb.make_star(0.2, sym[1]) if rot else qb.make_full_stadium(1.0, 1.0)
    make = qb.DLP_kress if rot else qb.DLP_kress_global_corners
    k = 5.0 + 0.03 * n
    pts, sol = qb.points_with_n(make(1.0, b, symmetry=_sym(qb, sym)), b, n, k)
    ws = qb.Workspace(sol, pts)
    ks = [k + 0.2j] if n == 128 else [k + 0.2j, k - 0.1 + 0.1j, k + 0.15 - 0.05j]
    panels = (6000, deg, 400, deg)
    ref = qb.assemble(ws, ks, cheb=panels) if deg == 5 else qb.assemble(ws, ks)
    out = qb.assemble(ws, ks, mixed=True, cheb=panels, split_lo=True)
    for q in range(len(ks)):
        v = out[q].astype(np.complex128) + out[len(ks) + q].astype(np.complex128)
        assert np.abs(v - ref[q]).max() <= 1e-13 * np.abs(ref[q]).max(), q
