"""General splines and graphs of every knot count through the batched kernels.

The lanes-over-points kernels find a dial's knot interval by halving steps, the
K = 1 kernels by five fixed steps; on the interval both do the same arithmetic.
Every event has one dial and its own bin, so a bin sum is that dial's response:
the 64-point sums must equal the one-point sums within the rounding of a few
operations, on the knots, between them and beyond the ends.
"""
import numpy as np
import pytest

from gundam_gb300 import _native as N
from gundam_gb300.engine import Engine

pytestmark = pytest.mark.gpu

KNOTS = (1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31)


def _engine(precision, k_max, truncate):
    rng = np.random.default_rng(12)
    dials = []
    for n in KNOTS:
        x = np.cumsum(rng.uniform(0.2, 1.0, n)).astype(np.float32).astype(np.float64) - 4.0
        y = rng.uniform(0.5, 1.5, n)
        dials.append((N.GW_DIAL_GRAPH, np.stack([y, x], 1).ravel()))
        if n > 1:
            dials.append((N.GW_DIAL_GENERAL, np.concatenate([[x[0], 1.0], np.stack([y, rng.normal(0, 0.3, n), x], 1).ravel()])))
    e = Engine(len(dials), 2, len(dials), k_max=k_max, precision=precision)
    if truncate:
        e.set_extrapolation(1, False)
    for p in (0, 1):
        e.set_lower_clamp(p, 0.0)
    e.set_event_indices(np.arange(len(dials), dtype=np.int32))
    for i, (t, d) in enumerate(dials):
        if t == N.GW_DIAL_GRAPH:
            e.add_graph(i, 1, d)
        else:
            e.add_spline(t, i, 1, d)
    e.set_data(np.ones(len(dials)))
    e.set_likelihood(N.GW_LLH_POISSON)
    e.initialize()
    return e, dials


@pytest.mark.parametrize("precision", ["fp32", "fp64", "df64"])
@pytest.mark.parametrize("truncate", [False, True])
def test_batched_interval_matches_one_point(precision, truncate):
    one, dials = _engine(precision, 1, truncate)
    many, _ = _engine(precision, 64, truncate)
    knots = np.concatenate([d[1::2] if t == N.GW_DIAL_GRAPH else d[4::3] for t, d in dials])
    rng = np.random.default_rng(5)
    pts = np.zeros((64, 2))
    pts[:40, 1] = rng.choice(knots, 40)  # on the knots, where the interval changes
    pts[40:, 1] = rng.uniform(-6.0, 16.0, 24)
    ref = np.concatenate([one.eval(pts[i:i + 1])[0] for i in range(64)])
    # a response is up to a dozen operations on values up to M: within 16 roundings of it
    eps = {"fp32": 2.0 ** -24, "fp64": 2.0 ** -53, "df64": 2.0 ** -44}[precision]
    scale = np.maximum(1.0, np.abs(ref)) * 100.0  # the cubic's terms beyond the ends cancel to the response
    tried = 0
    for i, (kind, ppp, _, _, _, _) in enumerate(Engine.compiled_shapes()):
        if kind != 0 or ppp > 64:
            continue
        try:
            many.set_shape_index(i)
        except RuntimeError:
            continue
        assert (np.abs(many.eval(pts)[0] - ref) <= 16 * eps * scale).all(), i
        tried += 1
    assert tried >= 2
    one.close()
    many.close()
