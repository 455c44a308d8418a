"""J0 and J1 near the origin relative to their own size (J1 ~ z / 2 vanishes
there beside Y1 ~ 1 / z, so a bound relative to both says nothing about it):
real arguments and the strip of the Taylor panels, across the change to the
power series at |z| = 0.25. Against SciPy's AMOS: the evaluator's 2e-14 plus as
much for AMOS."""
import numpy as np
import pytest
from scipy import special as sp

pytestmark = pytest.mark.gpu


def _check(qb, z):
    got = qb.bessel01(z)
    for c, ref in ((0, sp.jv(0, z)), (1, sp.jv(1, z))):
        err = np.abs(got[:, c] - ref) / np.abs(ref)
        assert err.max() <= 4e-14, (c, z[int(np.argmax(err))], err.max())


def test_real(qb):
    x = np.concatenate([10.0 ** np.linspace(-12, 0, 600)[:-1], [0.25, np.nextafter(0.25, 0), np.nextafter(0.25, 1), 0.999]])
    _check(qb, x.astype(complex))


@pytest.mark.parametrize("im", [1e-10, 1e-4, 0.01, 0.1, 0.2, 0.24, 0.25, 0.3, 0.4])
def test_strip(qb, im):
    x = np.concatenate([10.0 ** np.linspace(-8, 0, 300)[:-1], [np.sqrt(max(0.0625 - im * im, 1e-6))]])
    for s in (1, -1):
        _check(qb, x + 1j * s * im)
