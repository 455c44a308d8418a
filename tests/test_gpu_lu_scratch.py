"""Device bytes of FP64 factorisations: the operators and, per operator, what
grows with n only. The digits of one product (96 bytes for each of 128 n
elements) are the largest part of that; every later product of the stream
takes the same block, twice at most while sizes shrink. The allocator caches
what a call held, counted from an empty cache."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIGITS = 2 * 96 * 128        # bytes per row of an operator
INVERSES = 4 * 64 * 16       # of the diagonal blocks
MB = 1 << 20


def _held(qb, call):
    qb.release_cached_memory()
    call()
    return qb.pool_stats()["cached_bytes"]


@pytest.mark.parametrize("n", [768, 2048])
def test_bytes_of_fp64_operators(qb, n):
    c = qb.make_star(0.2, 5)
    k = 0.07 * n
    pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, n, k)
    ws = qb.Workspace(sol, pts)
    V = qb.probe_matrix(n, 32, np.random.default_rng(0))
    nq = 8

    def beyn():
        bh = qb.BeynHandle(ws, k, 0.3, nq, mixed=False)
        bh.moments(V)
        bh.close()

    vectors = 8 * 32 * 16    # right-hand sides, solutions and moments of 32 columns
    tables = 8 * MB          # 18000 panels of two series, with the rounding to 2 MB
    assert _held(qb, beyn) <= nq * (16 * n * n + (DIGITS + INVERSES + vectors) * n + tables)
    lanczos = 99 * 16
    for nk in (1, 8):
        got = _held(qb, lambda: qb.sigma_min(ws, list(k + 0.1 * np.arange(nk))))
        assert got <= nk * (16 * n * n + (DIGITS + INVERSES + lanczos) * n) + 16 * MB, nk


def test_two_threads_keep_their_blocks_apart(qb):
    from concurrent.futures import ThreadPoolExecutor
    c = qb.make_star(0.2, 5)
    made = []
    for n in (300, 404, 300, 404):
        pts, sol = qb.points_with_n(qb.CFIE_kress(1.0, c), c, n, 20.0)
        made.append(qb.Workspace(sol, pts))
    ks = [np.linspace(20.0, 20.4, 6 + q) for q in range(4)]
    alone = [qb.sigma_min(w, k) for w, k in zip(made, ks)]
    with ThreadPoolExecutor(4) as ex:
        for _ in range(3):
            for got, ref in zip(ex.map(qb.sigma_min, made, ks), alone):
                assert np.array_equal(got, ref)
