"""The Barlow-Beeston bin term next to one event, where the logarithms are small:
their error is relative, not absolute.  Without a sum of w^2 the term is
2 (p - d + d (log d - log p)); next to 1, p - d is exact.

Tolerance: each logarithm within 0.55 ulp, the other operations (the difference of
the logarithms, the fused product and sum; doublings are exact) half an ulp of
their results:
    2 (d (0.55 (ulp(log d) + ulp(log p)) + ulp(log d - log p) / 2) + ulp(term / 2) / 2).
"""
import numpy as np
import pytest

from gundam_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span", [0.1, 1e-2, 4e-3, 1e-4, 1e-7, 1e-11])
@pytest.mark.parametrize("data_is_one", [True, False])
def test_term_next_to_one_event(span, data_is_one):
    rng = np.random.default_rng(23)
    n = 1 << 15
    pred = 1 + rng.uniform(-span, span, n)
    data = np.ones(n) if data_is_one else 1 + rng.uniform(-span, span, n)
    got, sq = np.full(n, -1.0), np.zeros(n)
    assert N.libgw().gw_llh_bins(N.GW_LLH_BARLOW_BEESTON_OA2021, data.ctypes.data, pred.ctypes.data, sq.ctypes.data, n,
                                 got.ctypes.data) == N.GW_OK
    d, p = data.astype(np.longdouble), pred.astype(np.longdouble)
    ld, lp = np.log1p(d - 1), np.log1p(p - 1)
    half = p - d + d * (ld - lp)
    ulp = lambda a: np.where(a == 0, 0.0, np.spacing(np.abs(a.astype(np.float64))))  # noqa: E731
    wide = 8 * np.finfo(np.longdouble).eps * (abs(p - d) + d * (abs(ld) + abs(lp)))  # of the reference itself
    tol = 2 * (d * (0.55 * (ulp(ld) + ulp(lp)) + 0.5 * ulp(ld - lp)) + 0.5 * ulp(half)) + 2 * wide
    assert np.all(abs(got - 2 * half) <= tol), float((abs(got - 2 * half) / tol).max())
