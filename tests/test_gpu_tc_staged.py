"""Staged complex64 tensor-core products at the edges of their tiles (128 rows,
32 or up to 128 columns, 16 k a stage), with few CTAs (narrow tile) and many
(wide tile): against complex128, the bound of the other
complex64 product tests (4e-6 of |alpha| |A| |B| + |beta| |C|); and a NaN or an
infinity of an operand reaches exactly its row or column, also from the last
row or column, which the staging repeats past the operand's end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("M", [1, 127, 129])
@pytest.mark.parametrize("N,batch", [(1, 2), (31, 1), (33, 3), (33, 200), (90, 120), (128, 100), (130, 120), (300, 60)])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 32, 49])
def test_tile_edges(qb, M, N, batch, K):
    rng = np.random.default_rng([M, N, K])
    A, B, C0 = _rand(rng, (batch, M, K)), _rand(rng, (batch, K, N)), _rand(rng, (batch, M, N))
    got = qb.cgemm(A, B, C0, -0.5 + 1j, 0.25 - 2j, engine=2)
    A, B, C0 = (x.astype(np.complex128) for x in (A, B, C0))
    ref = (-0.5 + 1j) * (A @ B) + (0.25 - 2j) * C0
    bound = abs(-0.5 + 1j) * (np.abs(A) @ np.abs(B)) + abs(0.25 - 2j) * np.abs(C0)
    assert (np.abs(got - ref) <= 4e-6 * bound).all()


@pytest.mark.parametrize("M,N,K,batch", [(1153, 1281, 32, 2), (1153, 1281, 31, 2), (1280, 1152, 33, 2), (1290, 1280, 37, 1)])
def test_packed_and_staged_agree(qb, M, N, K, batch):
    rng = np.random.default_rng([M, K])
    A, B, C0 = _rand(rng, (batch, M, K)), _rand(rng, (batch, K, N)), _rand(rng, (batch, M, N))
    got, want = (qb.cgemm(A, B, C0, -1.0, 1.0, engine=e) for e in (1, 2))
    bound = np.abs(A) @ np.abs(B) + np.abs(C0)
    assert (np.abs(got - want) <= 2 * 4e-6 * bound).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("M,N,batch", [(128, 32, 1), (70, 21, 1), (130, 93, 160)])
def test_non_finite_stays_in_its_row_and_column(qb, bad, M, N, batch):
    rng = np.random.default_rng(3)
    A, B = _rand(rng, (batch, M, 20)), _rand(rng, (batch, 20, N))
    A[-1, M - 1, 3] = bad
    B[-1, 7, N - 1] = bad
    got = qb.cgemm(A, B, np.zeros((batch, M, N), np.complex64), 1.0, 0.0, engine=2)
    hit = np.zeros((batch, M, N), bool)
    hit[-1, M - 1] = hit[-1, :, N - 1] = True
    assert (np.isfinite(got) == ~hit).all()


@pytest.mark.parametrize("M,N,K", [(129, 130, 17), (300, 96, 256)])
def test_both_tile_widths_give_the_same_bits(qb, M, N, K):
    rng = np.random.default_rng(K)
    A, B, C0 = _rand(rng, (1, M, K)), _rand(rng, (1, K, N)), _rand(rng, (1, M, N))
    one = qb.cgemm(A, B, C0, -1.0, 1.0, engine=2)
    many = qb.cgemm(*(np.repeat(x, 100, axis=0) for x in (A, B, C0)), -1.0, 1.0, engine=2)
    assert (many == one).all()
