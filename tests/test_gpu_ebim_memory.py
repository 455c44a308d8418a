"""Device bytes of one EBIM eigen step: the three matrices, A^-1 A' and, for the
default form, nothing more of their size (the digit planes of the operator
take the factors' place): 80 n^2 bytes; the full form keeps its factors beside
the planes, 96 n^2; solve_vect 48 n^2. 64 MB for everything that grows with n only.
The allocator keeps a call's blocks, so what it caches after the call from an
empty cache is what the call held. Values against the window's own FP64
products (one column block below the digit products' size)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _held(qb, call):
    qb.release_cached_memory()
    before = qb.pool_stats()
    out = call()
    after = qb.pool_stats()
    assert after["live_bytes"] <= before["live_bytes"]
    return after["cached_bytes"] - before["cached_bytes"], out


@pytest.mark.parametrize("n", [1100, 2048])
@pytest.mark.parametrize("form,per", [("default", 80), ("full", 96), ("vect", 48)])
def test_bytes_held(qb, n, form, per):
    k = 0.07 * n
    if form == "vect":
        c = qb.make_circle(1.0)
        pts, sol = qb.points_with_n(qb.DLP_kress(1.0, c), c, n, k)
        ws = qb.Workspace(sol, pts)
        held, _ = _held(qb, lambda: qb.operators.solve_vect_dlp(ws, k))
    else:
        c = qb.make_circle_with_hole(1.0, (0.3, 0.1, 0.2))
        pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, n * 5 // 6 // 2 * 2, k)
        ws = qb.Workspace(sol, pts)
        held, _ = _held(qb, lambda: qb.ebim.solve(ws, k, 0.02, nev=5, full=form == "full"))
    m = ws.dim
    assert abs(m - n) <= 8
    assert held <= per * m * m + (64 << 20), (held - per * m * m) / 2.0 ** 20


def test_default_and_full_form_agree(qb):
    c = qb.make_circle_with_hole(1.0, (0.3, 0.1, 0.2))
    pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, 916, 70.0)
    ws = qb.Workspace(sol, pts)
    A, dA, ddA = qb.construct_matrices(sol, pts, ws, 70.0, derivs=True)
    eps = 16 * ws.dim * 2.0 ** -52 * np.linalg.cond(A) * np.linalg.norm(dA, 2)
    for full in (False, True):
        f = qb.ebim.solve_full if full else qb.ebim.solve_krylov
        ref = f(sol, A, dA, ddA, pts, 70.0, 0.02, nev=5, return_imag_part=True)[0]  # FP64 block iteration
        got = qb.ebim.solve(ws, 70.0, 0.02, nev=5, full=full, return_imag_part=True)[0]
        assert len(got) == len(ref) >= 1 and np.max(np.abs(np.sort_complex(got) - np.sort_complex(ref))) <= eps
