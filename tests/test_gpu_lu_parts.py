"""Mixed-form moments with one stream part and with four, on both sides of the
batch size from which parts are used (2.6e7 elements): bit-identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq", [(128, 8), (512, 99), (512, 101)])
def test_parts_bitwise_equal(qb, n, nq):
    b = qb.make_star(0.2, 5)
    pts, sol = qb.points_with_n(qb.DLP_kress(1.0, b), b, n, 20.0)
    ws = qb.Workspace(sol, pts)
    V = qb.probe_matrix(ws.dim, 24, np.random.default_rng(5))
    before, out = qb.autotune.lu_plan(), []
    try:
        for parts in (1, 4):
            qb.autotune.set_lu_plan(parts=parts)
            bh = qb.BeynHandle(ws, 20.0 + 0.05j, 0.4, nq, mixed=True)
            out.append(bh.moments(V))
            bh.close()
    finally:
        qb.autotune.set_lu_plan(**before)
    for a, r in zip(*out):
        assert np.array_equal(a, r)
