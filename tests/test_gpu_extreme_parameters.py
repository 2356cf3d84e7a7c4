"""Parameters that are no ordinary numbers, through every stored form of the splines
and every family of kernels."""
import numpy as np
import pytest

from gundam_gb300 import Engine
from gundam_gb300 import _native as N

pytestmark = pytest.mark.gpu

rng = np.random.default_rng(4)
X4, X3 = np.array([-3.0, -1.0, 0.0, 2.5]), np.array([-3.0, 0.5, 2.0])
Y = rng.uniform(0.5, 1.5, 16)
DIALS = [  # one event and one bin each; parameter 1 (and 2 for the surfaces)
    (N.GW_DIAL_NORM, np.zeros(0)),
    (N.GW_DIAL_MONOTONIC, np.concatenate([[-3.0, 1.0], Y[:7]])),
    (N.GW_DIAL_COMPACT, np.concatenate([[-3.0, 1.0], Y[:7]])),
    (N.GW_DIAL_UNIFORM, np.concatenate([[-3.0, 2.0], np.stack([Y[:4], rng.normal(0, 0.2, 4)], 1).ravel()])),
    (N.GW_DIAL_GENERAL, np.concatenate([[-3.0, 1.0], np.stack([Y[:4], rng.normal(0, 0.2, 4), X4], 1).ravel()])),
    (N.GW_DIAL_GRAPH, np.stack([Y[:4], X4], 1).ravel()),
    (N.GW_DIAL_BILINEAR, np.concatenate([[4, 3], X4, X3, Y[:12]])),
    (N.GW_DIAL_BICUBIC, np.concatenate([[4, 3], X4, X3, Y[:12]])),
]


def engine(precision, k_max, layout="auto", truncate=False, lo=None, hi=None):
    n = len(DIALS)
    e = Engine(n, 3, n, k_max=k_max, precision=precision, spline_layout=layout)
    for p in (1, 2):
        if truncate:
            e.set_extrapolation(p, False)
        if lo is not None:
            e.set_lower_clamp(p, lo)
        if hi is not None:
            e.set_upper_clamp(p, hi)
    e.set_event_indices(np.arange(n, dtype=np.int32))
    start = np.cumsum([0] + [d.size for _, d in DIALS]).astype(np.int64)
    e.add_dials(np.array([t for t, _ in DIALS], np.uint8), np.arange(n, dtype=np.int32), np.full(n, 1, np.int32),
                np.full(n, 2, np.int32), start, np.concatenate([d for _, d in DIALS]))
    e.set_data(np.ones(n))
    e.initialize()
    return e


def families(e, k):
    """Each family of kernels the engine has for k points (the first shape of each)."""
    if k == 1:
        for kind in (0, 1, 2):
            e.set_plain_kernel(kind)
            yield kind
        return
    done = set()
    for i, (kind, _, _, _, _, _) in enumerate(Engine.compiled_shapes()):
        if kind in done:
            continue
        try:
            e.set_shape_index(i)
        except RuntimeError:
            continue
        done.add(kind)
        yield kind
    assert len(done) >= 2


@pytest.mark.parametrize("precision", ["fp64", "fp32", "df64"])
@pytest.mark.parametrize("layout", ["auto", "knots", "slopes", "coefs", "grid"])
def test_nan_parameter(precision, layout):
    """NaN gives NaN in the bins of that point and nothing else."""
    for k in (1, 4, 24, 64):
        e = engine(precision, k, layout)
        pts = np.zeros((k, 3))
        pts[:, 1:] = np.linspace(-2.0, 1.5, k)[:, None]
        for _ in families(e, k):
            ref = e.eval(pts)[0]
            assert np.isfinite(ref).all()
            for sign in (1.0, -1.0):
                bad = pts.copy()
                bad[k // 2, 1:] = np.copysign(np.nan, sign)
                got = e.eval(bad)[0]
                assert np.isnan(got[k // 2]).all(), (k, got[k // 2])
                rest = np.arange(k) != k // 2
                assert np.array_equal(got[rest], ref[rest])
        e.close()


def _around(values):
    v = np.asarray(values, dtype=np.float64)
    with np.errstate(over="ignore"):
        return np.unique(np.concatenate([v, np.nextafter(v, np.inf), np.nextafter(v, -np.inf)]))


BOUNDS = [(None, None), (0.0, None), (-0.0, 1.0), (0.75, 1.25), (-1.5, -0.25), (-2.0, 0.0), (0.0, 0.0), (0.0, np.inf)]


@pytest.mark.parametrize("lo,hi", BOUNDS)
@pytest.mark.parametrize("k", [1, 64])
def test_fp64_clamp_at_its_bounds(k, lo, hi):
    """A norm dial's response is its parameter, so the clamp shows by itself: the same
    number as the comparisons v < lo and v > hi give."""
    big = np.finfo(np.float64).max
    edges = [0.0, 5e-324, 1.0, 1e20, 1e21, big] + [b for b in (lo, hi) if b is not None and np.isfinite(b)]
    vals = _around(edges + [-v for v in edges])
    vals = np.concatenate([vals, [-0.0, np.inf, -np.inf]])
    a, b = -big if lo is None else lo, big if hi is None else hi
    want = np.where(vals < a, a, np.where(vals > b, b, vals))
    e = engine("fp64", k, lo=lo, hi=hi)
    for _ in families(e, k):
        got = []
        for i in range(0, vals.size, k):
            pts = np.zeros((k, 3))
            pts[:vals[i:i + k].size, 1] = vals[i:i + k]
            got.append(e.eval(pts)[0][:vals[i:i + k].size, 0])
        assert np.array_equal(np.concatenate(got), want)
    e.close()


@pytest.mark.parametrize("layout", ["auto", "knots", "slopes", "coefs", "grid"])
@pytest.mark.parametrize("truncate", [False, True])
def test_fp64_responses_at_the_knots(layout, truncate):
    """On every knot, next to it and at both zeros (a knot of the surfaces' first axis
    is 0): the oracle's response.  A response between the ends is about sixteen
    operations on terms up to 8 (a cubic of unit values and slopes, its expansion
    about another origin); beyond the ends, three intervals out, the terms of the
    cubics reach 8 * 4^3.  The search picks either interval of a knot, where both
    give the knot's value."""
    from oracle import oracle as O

    x = np.concatenate([_around([-3.0, -2.0, -1.0, 0.0, 0.5, 1.0, 2.0, 2.5, 3.0]), [-0.0, 1e-300, -1e-300, 0.3, -1.7],
                        [-5.0, 6.0]])
    ends = [(t, *({N.GW_DIAL_GENERAL: (-3.0, 2.5), N.GW_DIAL_GRAPH: (-3.0, 2.5), N.GW_DIAL_BILINEAR: (-3.0, 2.0),
                   N.GW_DIAL_BICUBIC: (-3.0, 2.0), N.GW_DIAL_NORM: (-9.0, 9.0)}.get(t, (-3.0, 3.0)))) for t, _ in DIALS]
    if truncate:
        x = np.concatenate([x, [np.inf, -np.inf]])
    big = np.finfo(np.float64).max  # the clamp of a parameter without one
    want = np.clip([[O.dial(t, d, v, v, truncate) for t, d in DIALS] for v in x], -big, big)
    inside = np.array([[truncate or a <= v <= b for _, a, b in ends] for v in x])
    tol = 16 * 2.0 ** -53 * 8 * np.where(inside, 1.0, 4.0 ** 3)
    for k in (1, 4, 24, 64):
        e = engine("fp64", k, layout, truncate=truncate)
        for family in families(e, k):
            got = []
            for i in range(0, x.size, k):
                pts = np.zeros((k, 3))
                n = x[i:i + k].size
                pts[:n, 1:] = x[i:i + k, None]
                got.append(e.eval(pts)[0][:n])
            got = np.concatenate(got)
            for i in range(len(DIALS)):
                err = np.abs(got[:, i] - want[:, i]) / tol[:, i]
                assert err.max() <= 1.0, (k, family, DIALS[i][0], x[err.argmax()], err.max())
        e.close()
