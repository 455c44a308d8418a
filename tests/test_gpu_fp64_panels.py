"""FP64 LU with every panel form the cluster rule picks: one CTA per panel for
large batches, clusters of 2, 4, 8 and 16 CTAs for smaller ones, panels shorter
than the cluster has rows for, partial last panels and outer blocks. Explicit
inverses against the identity; the bound is eps times the condition number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inverse(A):
    from qbgpu import _lib as L
    batch, n, _ = A.shape
    a = np.ascontiguousarray(A.transpose(0, 2, 1))
    x = np.empty_like(a)
    L.check(L.load().qbg_dense_inverse(n, batch, 0, L.vptr(a), L.vptr(x), None, None))
    return x.transpose(0, 2, 1)


@pytest.mark.parametrize("n,batch", [(1, 1), (2, 3), (5, 160), (33, 1), (65, 16), (97, 40), (130, 77), (200, 153), (259, 20), (515, 9), (1030, 2)])
def test_inverse(qb, n, batch):
    rng = np.random.default_rng(n + batch)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)) + 2.0 * np.sqrt(n) * np.eye(n)[rng.permutation(n)]
    X = _inverse(A)
    for b in sorted({0, batch // 2, batch - 1}):
        cond = np.linalg.cond(A[b])
        assert np.linalg.norm(A[b] @ X[b] - np.eye(n)) <= 2e-15 * n * cond, b
