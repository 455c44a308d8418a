"""Device Bessel functions at the edges of their ranges: the unit Taylor panels
(real argument; |Im z| <= 0.4), the change from G0 to Y0 at Re z = 6, the end of
the panels at 128, the fixed asymptotic sums from |z| = 32 and 128, and the
general routines outside the strip. Against SciPy's AMOS; the bound is the
evaluator's 2e-14 plus as much for AMOS, relative to max(|J|, |Y|)."""
import numpy as np
import pytest
from scipy import special as sp

pytestmark = pytest.mark.gpu

EDGES = [1e-8, 1e-3, 0.5, 1.0, 2.0, 5.0, 6.0, 7.0, 14.5, 25.0, 32.0, 64.0, 127.0, 128.0, 129.0, 500.0, 1700.0]


def _check(qb, z):
    got = qb.bessel01(z)
    ref = np.stack([sp.jv(0, z), sp.jv(1, z), sp.yv(0, z), sp.yv(1, z)], axis=1)
    for a, b in ((0, 2), (1, 3)):
        scale = np.maximum(np.abs(ref[:, a]), np.abs(ref[:, b]))
        for c in (a, b):
            err = np.abs(got[:, c] - ref[:, c]) / scale
            # the argument's own rounding: half an ulp of |z| in the phase
            bound = 4e-14 + np.abs(z) * 2.3e-16
            worst = int(np.argmax(err / bound))
            assert err[worst] <= bound[worst], (z[worst], c, err[worst])


def test_real_arguments(qb):
    x = np.concatenate([[e, np.nextafter(e, 0.0), np.nextafter(e, 1e9), e * 0.999, e * 1.001] for e in EDGES])
    rng = np.random.default_rng(5)
    x = np.concatenate([x, rng.uniform(1e-3, 200.0, 4000)])
    got = qb.bessel01(x.astype(complex))
    assert np.all(got.imag == 0.0)
    _check(qb, x.astype(complex))


@pytest.mark.parametrize("im", [1e-9, 0.01, 0.4, 0.4000001, 0.49, 0.51, 1.0, 2.5])
def test_complex_arguments(qb, im):
    x = np.concatenate([[e, e * 0.999, e * 1.001] for e in EDGES if e >= 0.5])
    rng = np.random.default_rng(6)
    x = np.concatenate([x, rng.uniform(0.3, 200.0, 1000)])
    _check(qb, x + 1j * im)
    lo, hi = qb.bessel01(x - 1j * im), qb.bessel01(x + 1j * im)
    scale = np.abs(hi).max(axis=1, keepdims=True)
    assert np.all(np.abs(lo - hi.conj()) <= 4e-15 * scale + 1e-300)


def test_non_finite_arguments_stay_non_finite(qb):
    got = qb.bessel01(np.array([np.nan, complex(np.nan, 0.1), complex(10.0, np.nan)]))
    assert np.all(np.isnan(got.real) | np.isnan(got.imag))
