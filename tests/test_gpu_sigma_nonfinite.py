"""sigma_min of operators with entries that are not finite: NaN, never the 0 of an
exactly singular operator, which a sweep would take for an eigenvalue. The
boundary's weights carry the NaN or the infinity into one column (at the start,
inside and at the end of a panel), for operators of one block and of several,
alone and in a batch; an operator without them keeps its value."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workspace(qb, n, at=None, value=0.0):
    c = qb.make_circle(1.0)
    pts, sol = qb.points_with_n(qb.DLP_kress(1.0, c), c, n, 0.08 * n)
    if at is not None:
        w = pts.ws.copy()
        w[at] = value
        pts = dataclasses.replace(pts, ws=w)
    return qb.Workspace(sol, pts)


@pytest.mark.parametrize("n", [40, 130])
@pytest.mark.parametrize("nk", [1, 40])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(qb, n, nk, bad):
    ks = 0.08 * n + 0.01 * np.arange(nk)
    for at in (0, n // 2, n - 1):
        assert np.all(np.isnan(qb.sigma_min(_workspace(qb, n, at, bad), ks))), at
    sig = qb.sigma_min(_workspace(qb, n), ks)
    assert np.all(sig > 0.0) and np.all(np.isfinite(sig))
