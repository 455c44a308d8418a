"""Matrices handed in by a caller, with rows scaled over 24 decades: the FP64
LU has to treat every row to its own magnitude. The scales are powers of two,
so A = D B differs from B by its pivot order only: the inverse is B^-1 D^-1, and
the pencil (D B, D B') has the eigenpairs and left vectors (up to D^-1) of
(B, B'). Bound: n eps cond(B), with 16 for the two factorisations' constants;
for the pencil beside what LAPACK's elimination loses to the pivot order."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _scales(n, rng):
    return 2.0 ** rng.permutation(np.round(-80.0 * np.arange(n) / n))


@pytest.mark.parametrize("n,batch", [(48, 1), (96, 3), (200, 1), (280, 2)])
def test_inverse_of_row_scaled_matrices(qb, n, batch):
    from qbgpu import _lib as L
    rng = np.random.default_rng(n)
    B = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)) + 2.0 * np.sqrt(n) * np.eye(n)
    d = _scales(n, rng)
    a = np.ascontiguousarray((d[:, None] * B).transpose(0, 2, 1))
    x = np.empty_like(a)
    L.check(L.load().qbg_dense_inverse(n, batch, L.QBG_PREC_FP64, L.vptr(a), L.vptr(x), None, None))
    X = x.transpose(0, 2, 1) * d  # A^-1 D
    for b in range(batch):
        ref = np.linalg.inv(B[b])
        assert np.linalg.norm(X[b] - ref) <= 16 * n * EPS * np.linalg.cond(B[b]) * np.linalg.norm(ref), b


def _full(A, dA, ddA, k, dk):
    """solve_full! in LAPACK's FP64: eigenpairs of A^-1 A', left vectors A^-H u."""
    mu, u, v = sl.eig(np.linalg.solve(A, dA), left=True)
    u = np.linalg.solve(A.conj().T, u)
    out = []
    for j in np.argsort(-np.abs(mu)):
        lam = 1.0 / mu[j]
        if abs(lam.real) < dk and abs(lam.imag) < dk:
            out.append(k - lam - 0.5 * lam * lam * (u[:, j].conj() @ ddA @ v[:, j]) / (u[:, j].conj() @ dA @ v[:, j]))
    return np.sort_complex(np.array(out))


@pytest.mark.parametrize("n", [50, 96, 200])
def test_ebim_of_a_row_scaled_pencil(qb, n):
    rng = np.random.default_rng(n + 1)
    A, dA, ddA = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))
    A = A + 1.5 * np.sqrt(n) * np.eye(n)
    d = _scales(n, rng)[:, None]
    k, dk = 10.0, 1.2
    ref = _full(A, dA, ddA, k, dk)
    lapack = np.max(np.abs(_full(d * A, d * dA, d * ddA, k, dk) - ref))
    got = np.sort_complex(qb.ebim.solve_full(None, d * A, d * dA, d * ddA, None, k, dk, return_imag_part=True)[0])
    assert 3 <= len(ref) < n // 2 and len(got) == len(ref)
    # as near as FP64 elimination of the same scaled matrices comes: its error here, or the unscaled pencil's
    assert np.max(np.abs(got - ref)) <= 32 * lapack + 16 * n * EPS * np.linalg.cond(A) * np.linalg.norm(dA, 2)
