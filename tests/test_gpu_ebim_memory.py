"""Device bytes of one EBIM eigen step: the three matrices, A^-1 A' and, for the
default form, nothing more of their size (the digit planes of the operator
take the factors' place): 80 n^2 bytes; the full form keeps its factors beside
the planes, 96 n^2; solve_vect 48 n^2. Beside that what grows with n: the digits
of a product of the factorisation (twice, while sizes shrink), the inverses of
the diagonal blocks, and the vectors of the block iteration. The allocator
keeps a call's blocks, so what it caches after the call from an empty cache is
what the call held. Then the values, with the block iteration's products from
digits, against those of the same matrices handed in, which stay in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _held(qb, call):
    qb.release_cached_memory()
    call()
    return qb.pool_stats()["cached_bytes"]


def _linear(n, nev=5, blocks=2):
    p = 2 * nev + 12
    digits, inverses = 2 * 96 * 128 * n, 4 * 64 * 16 * n
    vectors = blocks * 16 * n * p * (4 + 16)  # two iterations: Q, Y, W, V and up to 16 partial products
    return digits + inverses + vectors + 32 * (2 << 20)  # some 30 blocks rounded up to 2 MB


@pytest.mark.parametrize("n", [2048, 3072])
@pytest.mark.parametrize("form,per", [("default", 80), ("full", 96), ("vect", 48)])
def test_bytes_held(qb, n, form, per):
    k = 0.07 * n
    if form == "vect":
        c = qb.make_circle(1.0)
        pts, sol = qb.points_with_n(qb.DLP_kress(1.0, c), c, n, k)
        ws = qb.Workspace(sol, pts)
        held = _held(qb, lambda: qb.operators.solve_vect_dlp(ws, k))
    else:
        c = qb.make_circle_with_hole(1.0, (0.3, 0.1, 0.2))
        pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, round(n / 2.4) * 2, k)
        ws = qb.Workspace(sol, pts)
        held = _held(qb, lambda: qb.ebim.solve(ws, k, 0.02, nev=5, full=form == "full"))
    m = ws.dim
    assert abs(m - n) <= 8
    assert held <= per * m * m + _linear(m), (held - per * m * m) / 2.0 ** 20


@pytest.mark.parametrize("full", [False, True])
def test_digits_against_fp64_products(qb, full):
    c = qb.make_circle_with_hole(1.0, (0.3, 0.1, 0.2))
    k, dk = 70.0, 0.05
    pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, 916, k)
    ws = qb.Workspace(sol, pts)
    A, dA, ddA = qb.construct_matrices(sol, pts, ws, k, derivs=True)
    eps = 16 * ws.dim * 2.0 ** -52 * np.linalg.cond(A) * np.linalg.norm(dA, 2)
    f = qb.ebim.solve_full if full else qb.ebim.solve_krylov
    ref = np.sort_complex(f(sol, A, dA, ddA, pts, k, dk, nev=5, return_imag_part=True)[0])
    got = np.sort_complex(qb.ebim.solve(ws, k, dk, nev=5, full=full, return_imag_part=True)[0])
    assert len(got) == len(ref) >= 1 and np.max(np.abs(got - ref)) <= eps
