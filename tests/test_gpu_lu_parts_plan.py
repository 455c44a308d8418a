"""The number of stream parts that a caller sets is the number a Beyn handle
uses, for small batches too: every part launches its own chain of kernels, so
the launches of a handle's creation grow with the parts. The default (-1) keeps
a small batch on one stream, and reading and setting the plan restores it. The
tuner tries the part counts for complex64 only, and its clusters in FP64 only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(qb, ws, parts, nq=8):
    qb.autotune.set_lu_plan(parts=parts)
    V = qb.probe_matrix(ws.dim, 16, np.random.default_rng(5))
    a = qb.launch_count()
    bh = qb.BeynHandle(ws, 20.0 + 0.05j, 0.4, nq, mixed=True)
    out = bh.moments(V)
    bh.close()
    return qb.launch_count() - a, out


@pytest.mark.parametrize("n", [128, 512])
def test_small_batches_take_the_parts_set(qb, n):
    b = qb.make_star(0.2, 5)
    pts, sol = qb.points_with_n(qb.DLP_kress(1.0, b), b, n, 20.0)
    ws = qb.Workspace(sol, pts)
    before = qb.autotune.lu_plan()
    try:
        got = {p: _launches(qb, ws, p) for p in (1, 2, 4, -1)}
        assert qb.autotune.lu_plan()["parts"] == -1
        qb.autotune.set_lu_plan(outer=before["outer"])
        assert qb.autotune.lu_plan()["parts"] == -1
    finally:
        qb.autotune.set_lu_plan(**before)
    assert got[1][0] < got[2][0] < got[4][0]
    assert got[-1][0] == got[1][0]
    for p in got:
        for x, y in zip(got[p][1], got[1][1]):
            assert np.array_equal(x, y), p


@pytest.mark.parametrize("mixed", [True, False])
def test_tuner_leaves_out_plans_that_run_alike(qb, mixed):
    b = qb.make_star(0.2, 5)
    pts, sol = qb.points_with_n(qb.DLP_kress(1.0, b), b, 128, 12.0)
    ws = qb.Workspace(sol, pts)
    before = qb.autotune.lu_plan()
    try:
        qb.autotune.set_lu_plan(parts=-1)
        best = qb.autotune.tune_beyn(sol, pts, ws, 12.0, 0.3, 8, 12, mixed=mixed, reps=1)
    finally:
        qb.autotune.set_lu_plan(**before)
    if mixed:
        assert [t["parts"] for t in best["table"][:4]] == [-1, 2, 4, 8]
        assert all(t["cluster"] != 1 for t in best["table"])
    else:
        assert all(t["parts"] == -1 for t in best["table"])
