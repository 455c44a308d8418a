"""The reduced DLP in the mixed form with coarse Chebyshev panels. Its terms are
image kernels, which on the H and J tables saw the H panels only, so neither few
J panels nor a high degree on wide ones may lower its accuracy: double-float
words hi + lo against the FP64 direct assembly, within the 1e-13 of the max-norm
that holds for panels resolved beyond rounding. Real and complex wavenumbers,
one chunk of contour nodes and several disks; panels that the tuner comes to at
1e-8, and a J count far below the H count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,panels", [(500, 35.0, (300, 10, 60, 10)), (2048, 150.0, (1520, 9, 305, 9)),
                                        (2048, 150.0, (1520, 10, 203, 10)), (2048, 150.0, (6000, 9, 60, 9)),
                                        (500, 35.0, (6000, 7, 40, 7)), (500, 35.0, (2000, 16, 4, 16))])
@pytest.mark.parametrize("sym", ["x", "xy"])
def test_coarse_panels(qb, n, k, panels, sym):
    b = qb.make_full_stadium(1.0, 1.0)
    s = qb.XReflection(-1) if sym == "x" else qb.XYReflection(-1, 1)
    pts, sol = qb.points_with_n(qb.DLP_kress_global_corners(1.0, b, symmetry=s), b, n, k)
    ws = qb.Workspace(sol, pts)
    ks = [k + 0.05j, k - 0.3 + 0.02j, k]
    ref = qb.assemble(ws, ks)
    out = qb.assemble(ws, ks, mixed=True, cheb=panels, split_lo=True)
    for q in range(len(ks)):
        v = out[q].astype(np.complex128) + out[len(ks) + q].astype(np.complex128)
        assert np.abs(v - ref[q]).max() <= 1e-13 * np.abs(ref[q]).max(), q


def test_beyn_with_coarse_panels(qb):
    b = qb.make_full_stadium(1.0, 1.0)
    k = 60.0
    pts, sol = qb.points_with_n(qb.DLP_kress_global_corners(1.0, b, symmetry=qb.XYReflection(-1, -1)), b, 800, k)
    ws = qb.Workspace(sol, pts)
    V = qb.probe_matrix(ws.dim, 24, np.random.default_rng(0))
    got = []
    for panels in ((6000, 9, 40, 9), (6000, 9, 3000, 9)):
        h = qb.BeynHandle(ws, [k, k + 0.7], [0.3, 0.3], 12, mixed=True, cheb=panels)
        got.append(h.moments(V)[0])
        h.close()
    # both panel sets resolve the operator to rounding: 1e-13 of it, times the conditioning of the solves
    assert np.abs(got[0] - got[1]).max() <= 1e-10 * np.abs(got[1]).max()
