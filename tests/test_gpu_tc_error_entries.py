"""A tensor-core product that gave up writes nothing and sets the sticky device
flag; every entry whose FP64 LU or solves run such products must then report
QBG_ECUDA instead of returning what the buffers held. The flag is set by one
product under a poll limit of 0, with the limit restored before the entries
run. After the flag is cleared the entries give their earlier results again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _entries(qb):
    from qbgpu import _lib as L
    rng = np.random.default_rng(3)
    n = 200
    A = np.asfortranarray(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 30.0 * np.eye(n))

    def inverse():
        X = np.empty_like(A)
        L.check(L.load().qbg_dense_inverse(n, 1, L.QBG_PREC_FP64, L.vptr(A), L.vptr(X), None, None))
        return X

    c = qb.make_circle(1.0)
    pts, sol = qb.points_with_n(qb.DLP_kress(1.0, c), c, 200, 12.0)
    ws = qb.Workspace(sol, pts)
    cs = qb.make_star(0.2, 5)
    pc, sc = qb.points_with_n(qb.CFIE_kress(1.0, cs), cs, 200, 12.0)
    wc = qb.Workspace(sc, pc)
    V = qb.probe_matrix(wc.dim, 16, np.random.default_rng(5))

    def beyn():
        bh = qb.BeynHandle(wc, 12.0, 0.3, 8, mixed=False)
        try:
            return np.stack(bh.moments(V))
        finally:
            bh.close()

    return dict(inverse=inverse, newton=lambda: np.array(qb.newton_refine_svd(wc, 12.0, 11.9, 12.1)),
                vect=lambda: qb.operators.solve_vect_dlp(ws, 12.0)[1], sweep=lambda: qb.sigma_min(wc, [12.0, 12.1]),
                ebim=lambda: np.array(qb.ebim.solve(wc, 12.0, 0.2, nev=3)), beyn=beyn)


@pytest.mark.parametrize("name", ["inverse", "newton", "vect", "sweep", "ebim", "beyn"])
def test_entry_reports_a_product_that_gave_up(qb, name):
    from qbgpu import _lib as L
    lib = L.load()
    call = _entries(qb)[name]
    before = call()
    a = np.ones((256, 256), np.complex64)
    try:
        L.check(lib.qbg_set_tc_wait_limit(0))
        with pytest.raises(L.QBGError):
            qb.cgemm(a, a)
        L.check(lib.qbg_set_tc_wait_limit(-1))
        with pytest.raises(L.QBGError) as ei:
            call()
        assert ei.value.status == L.QBG_ECUDA and "gave up" in str(ei.value)
    finally:
        lib.qbg_set_tc_wait_limit(-1)
        lib.qbg_clear_tc_error()
    assert np.array_equal(call(), before)
