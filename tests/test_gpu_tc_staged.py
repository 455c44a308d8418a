"""Staged complex64 tensor-core products at the edges of their tiles (128 rows,
32 columns, 16 k a stage): against complex128, the bound of the other
complex64 product tests (4e-6 of |alpha| |A| |B| + |beta| |C|); and a NaN or an
infinity of an operand reaches exactly its row or column, also from the last
row or column, which the staging repeats past the operand's end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("M", [1, 127, 129])
@pytest.mark.parametrize("N,batch", [(1, 2), (31, 1), (33, 3)])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 32, 49])
def test_tile_edges(qb, M, N, batch, K):
    rng = np.random.default_rng([M, N, K])
    A, B, C0 = _rand(rng, (batch, M, K)), _rand(rng, (batch, K, N)), _rand(rng, (batch, M, N))
    got = qb.cgemm(A, B, C0, -0.5 + 1j, 0.25 - 2j, engine=2)
    A, B, C0 = (x.astype(np.complex128) for x in (A, B, C0))
    ref = (-0.5 + 1j) * (A @ B) + (0.25 - 2j) * C0
    bound = abs(-0.5 + 1j) * (np.abs(A) @ np.abs(B)) + abs(0.25 - 2j) * np.abs(C0)
    assert (np.abs(got - ref) <= 4e-6 * bound).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("M,N", [(128, 32), (70, 21)])
def test_non_finite_stays_in_its_row_and_column(qb, bad, M, N):
    rng = np.random.default_rng(3)
    A, B = _rand(rng, (M, 20)), _rand(rng, (20, N))
    A[M - 1, 3] = bad
    B[7, N - 1] = bad
    got = qb.cgemm(A, B, np.zeros((M, N), np.complex64), 1.0, 0.0, engine=2)
    hit = np.zeros((M, N), bool)
    hit[M - 1] = hit[:, N - 1] = True
    assert (np.isfinite(got) == ~hit).all()
