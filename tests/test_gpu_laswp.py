"""Row interchanges of the LU panels: solutions of systems whose pivots come in every
order (reversed rows, rotated rows, a random permutation, no interchange at all),
at sizes below, at and off the panel width and with a batch, complex64 and complex128.
The matrices are permutations plus a perturbation of 1e-2 / n, so the condition
number is below 1.1 and the inverse is good to a few roundings: 1e-13 and 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 65, 96, 127, 129, 200, 513])
@pytest.mark.parametrize("order", ["none", "reversed", "rotated", "random"])
@pytest.mark.parametrize("single,tol", [(False, 1e-13), (True, 1e-5)])
def test_inverse_of_permutations(qb, n, order, single, tol):
    from qbgpu import _lib as L
    rng = np.random.default_rng([n, len(order)])
    perm = {"none": np.arange(n), "reversed": np.arange(n)[::-1], "rotated": np.roll(np.arange(n), 33),
            "random": rng.permutation(n)}[order]
    A = np.zeros((2, n, n), complex)
    A[0, np.arange(n), perm] = 1.0
    A[1, perm, np.arange(n)] = 1j
    A += 1e-2 / n * (rng.uniform(-1, 1, A.shape) + 1j * rng.uniform(-1, 1, A.shape))
    a = np.ascontiguousarray(A.transpose(0, 2, 1))
    X = np.empty_like(a)
    L.check(L.load().qbg_dense_inverse(n, 2, L.QBG_PREC_FP32 if single else 0, L.vptr(a), L.vptr(X), None, None))
    for q in range(2):
        assert np.abs(X[q].T @ A[q] - np.eye(n)).max() <= tol
