"""complex128 products on the tensor cores at the sizes the FP64 LU's short
products have: one pass per operand up to K = 128, two above; rows, k and
columns at and around the 16, 32 and 128 tiles; the bound of the other
products, 4e-15 (|A| |B|) + 2^-52 |C'| elementwise. Rows and columns holding
Inf or NaN give NaN there and nowhere else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [16, 31, 33, 128, 130])
@pytest.mark.parametrize("N", [16, 31, 33])
@pytest.mark.parametrize("K", [16, 23, 32, 120, 127, 128, 129])
def test_small_products_vs_exact(qb, M, N, K):
    rng = np.random.default_rng(M * 10007 + N * 101 + K)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    A, B, C = z(3, M, K), z(3, K, N), z(3, M, N)
    ld = np.clongdouble
    ref = C.astype(ld) - A.astype(ld) @ B.astype(ld)
    allowed = 4e-15 * (np.abs(A) @ np.abs(B)) + 2.0 ** -52 * np.abs(ref).astype(np.float64)
    err = np.abs(qb.zgemm_sub_tc(A, B, C).astype(ld) - ref).astype(np.float64)
    assert np.max(err / allowed) <= 1.0


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_stay_in_their_row_and_column(qb, bad):
    rng = np.random.default_rng(4)
    A, B, C = (rng.standard_normal(s) + 1j * rng.standard_normal(s) for s in ((40, 32), (32, 35), (40, 35)))
    A[7, 3], B[5, 30] = bad, complex(0.0, bad)
    out = qb.zgemm_sub_tc(A, B, C)
    hit = np.zeros((40, 35), bool)
    hit[7, :] = True
    hit[:, 30] = True
    assert np.all(np.isnan(out.real[hit]) & np.isnan(out.imag[hit]))
    assert np.all(np.isfinite(out[~hit]))


@pytest.mark.parametrize("n,nrhs", [(20, 5), (31, 1), (33, 16), (96, 17), (161, 64), (290, 70)])
def test_fp64_solves_of_every_block_form(qb, n, nrhs):
    """The FP64 LU and solves through a Beyn handle's moments: sizes below, at
    and off the 32-row blocks, right-hand sides below and above 16 columns,
    against LAPACK on the same operators (backward-stable on both sides)."""
    b = qb.make_star()
    pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, b), b, n + n % 2, 0.1 * n)
    ws = qb.Workspace(sol, pts)
    rng = np.random.default_rng(n)
    V = np.asfortranarray(rng.standard_normal((ws.dim, nrhs)) + 1j * rng.standard_normal((ws.dim, nrhs)))
    k0, R, nq = max(2.0, 0.1 * n), 0.4, 5
    bh = qb.BeynHandle(ws, k0, R, nq, use_chebyshev=False)
    A0, A1 = bh.moments(V)
    bh.close()
    zj, wj = qb.contour(k0, R, nq)
    T = qb.assemble(ws, zj)
    X = [np.linalg.solve(t, V) for t in T]
    cond = max(np.linalg.cond(t) for t in T)
    for A, w in ((A0, wj), (A1, wj * zj)):
        scale = sum(abs(a) * np.linalg.norm(x) for a, x in zip(w, X))
        ref = sum(a * x for a, x in zip(w, X))
        assert np.linalg.norm(A - ref) <= 1e-14 * cond * scale
