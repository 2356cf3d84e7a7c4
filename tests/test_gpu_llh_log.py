"""The Barlow-Beeston bin term where only its logarithm and its clamps work (no
sum of w^2: 2 (p - d + d (log d - log p))), against extended precision.

Tolerance: the logarithms are good to 0.75 ulp (2e-18 near 1) and each of the
other operations to half an ulp of its result, with u = 2^-52:
    2 (u (d + p) + d (u (|log d| + |log p| + |log d - log p|) + 4e-18)) + 2 u |term|.
Predictions at or below the smallest normal double enter as that number; equal
data and prediction give exactly zero."""
import numpy as np
import pytest

from gundam_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _terms(data, pred):
    out = np.full(data.size, -1.0)
    sq = np.zeros(data.size)
    assert N.libgw().gw_llh_bins(N.GW_LLH_BARLOW_BEESTON_OA2021, data.ctypes.data, pred.ctypes.data, sq.ctypes.data,
                                 data.size, out.ctypes.data) == N.GW_OK
    return out


@pytest.mark.parametrize("span", ["exponents", "binade", "close"])
def test_term_without_uncertainty(span):
    rng = np.random.default_rng(17)
    n = 1 << 16
    if span == "exponents":
        data, pred = 10.0 ** rng.uniform(-15, 15, n), 10.0 ** rng.uniform(-307, 15, n)
        pred[:4] = [np.finfo(float).tiny, 5e-324, 2 * np.finfo(float).tiny, 0.0]
    elif span == "binade":
        data, pred = rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n)
    else:
        data = 10.0 ** rng.uniform(-3, 6, n)
        pred = data * (1 + rng.uniform(-1e-6, 1e-6, n))
    got = _terms(data, pred)
    d, p = data.astype(np.longdouble), np.maximum(pred, np.finfo(float).tiny).astype(np.longdouble)
    ld, lp = np.log(d), np.log(p)
    ref = 2 * (p - d + d * (ld - lp))
    u = 2.0 ** -52
    tol = 2 * (u * (d + p) + d * (u * (abs(ld) + abs(lp) + abs(ld - lp)) + 4e-18)) + 2 * u * abs(ref)
    assert np.all(abs(got - ref) <= tol), float((abs(got - ref) / tol).max())
    assert np.all(_terms(data, data.copy()) == 0.0)
