"""The surrogate's head kernels and GEMM tile choices at the edges of their ranges.

* An additive base of few nodes goes through the staged kernels; the same
  piecewise-linear functions written on a refined node grid go through the
  general ones.  Both must agree within FP32 rounding.
* The GEMM's tile shapes, chosen by size, against an FP64 product.
"""
import numpy as np
import pytest

from gundam_gb300 import _native as N
from gundam_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _surrogate(P, B, nodes, refine, seed, ratio):
    """An additive surrogate with a zero network; refine: each interval cut into that many equal ones."""
    rng = np.random.default_rng(seed)
    s = Surrogate(P, B, hidden=(8,), batch_max=128, seed=1)
    s.mlp.set_layer(1, np.zeros((B, 8), np.float32), np.zeros(B, np.float32))
    tab = rng.normal(0, 0.05, (P, nodes, B)).astype(np.float32).astype(np.float64)
    fine = (nodes - 1) * refine + 1
    at = np.arange(fine) / refine
    i = np.minimum(at.astype(int), nodes - 2)
    t = (at - i)[None, :, None]
    tab = tab[:, i] * (1 - t) + tab[:, i + 1] * t
    s.kind, s.nodes, s.lim = "additive", fine, 3.0
    s.mu, s.sd = np.zeros(P), np.ones(P)
    s.A = np.concatenate([rng.uniform(3.0, 5.0, (1, B)), tab.reshape(P * fine, B)])
    s.r_mu, s.r_sd = np.zeros(B), np.full(B, 0.01)
    s.rb, s.rw = rng.normal(0, 0.1, B), (rng.normal(0, 0.05, (B, P)) if ratio else np.zeros((B, P)))
    data = rng.poisson(np.exp(s.A[0])).astype(np.float64)
    s.attach(data, None if ratio else np.exp(s.rb), N.GW_LLH_BARLOW_BEESTON_OA2021)
    return s, data


@pytest.mark.parametrize("P,B,nodes,C,ratio", [(8, 8, 2, 1, True), (16, 64, 8, 8, True), (24, 72, 5, 9, False),
                                               (200, 264, 8, 65, True), (48, 520, 7, 128, True)])
def test_staged_head_matches_the_general_form(P, B, nodes, C, ratio):
    theta = np.random.default_rng(P + C).normal(0, 1.5, (C, P))  # beyond the outer nodes too
    staged, data = _surrogate(P, B, nodes, 1, 3, ratio)
    general, _ = _surrogate(P, B, nodes, 8, 3, ratio)
    assert staged.nodes <= 8 < general.nodes
    l0, r0 = staged.device_log_rates(theta)
    l1, r1 = general.device_log_rates(theta)
    # a log rate is a sum of P interpolations of values up to T about b0 <= 5: each term and each
    # partial sum rounded, and the refined nodes rounded once more
    T = np.abs(staged.A[1:]).max()
    delta = EPS * (P * (5 + P * T) + 8 * P * T)
    assert np.abs(r0 - r1).max() <= delta
    # d term / d log rate is at most 2 (2 mu + n): the terms' own FP32 rounding beside it
    mu = np.exp(r0)
    reach = (4 * mu + 2 * data).sum(axis=1)
    assert (np.abs(l0 - l1) <= reach * (2 * delta + 64 * EPS)).all()
    f0, g0 = staged.value_grad(theta)
    f1, g1 = general.value_grad(theta)
    assert (np.abs(f0 - f1) <= reach * (2 * delta + 64 * EPS)).all()
    # the refined slopes are differences of values up to T over an eighth of the step; G and S move by
    # at most 8 mu per unit of log rate, and every product and sum over the bins is rounded
    step = 6.0 / (nodes - 1)
    slope = 2 * T / step + 0.3
    tol = (reach * (2 * EPS * T * 8 / step) + 8 * mu.sum(axis=1) * (2 * delta + 64 * EPS) * slope
           + reach * slope * 32 * EPS)
    # a point within rounding of a node may take the slope of either side
    u = (np.clip(theta, -3, 3) + 3.0) / step
    off_node = np.abs(u - np.round(u)) > 1e-5
    assert (np.abs(g0 - g1)[off_node] <= np.broadcast_to(tol[:, None], g0.shape)[off_node]).all()
    staged.close()
    general.close()


def _bits(x):
    b = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
    return ((b + 0x7FFF + ((b >> 16) & 1)) >> 16).astype(np.uint16)


# one row or one short tile; more K steps than stages; columns that are no multiple of a vector;
# then the sizes at which 64-, 128- and 256-column tiles are chosen
@pytest.mark.parametrize("M,N_,K", [(8, 32, 8), (1, 8, 16), (64, 3000, 520), (129, 33, 1032), (200, 250, 64),
                                    (1216, 520, 136), (2432, 1048, 72), (2432, 2056, 72)])
def test_gemm_tile_choices(M, N_, K):
    import ctypes as C
    rng = np.random.default_rng(M + N_ + K)
    a16, b16 = _bits(rng.standard_normal((M, K))), _bits(rng.standard_normal((N_, K)))
    out = np.full((M, N_), np.nan, np.float32)
    p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert N.libgw().gwm_gemm_test(p(a16), p(b16), M, N_, K, p(out)) == 0
    wide = lambda x: (x.astype(np.uint32) << 16).view(np.float32).astype(np.float64)  # noqa: E731
    ref = wide(a16) @ wide(b16).T
    # FP32 accumulation: K roundings of partial sums of size ~ sqrt(K), with room for the tail
    assert (np.abs(out - ref) <= 8 * EPS * np.sqrt(K) * (np.sqrt(K) + np.abs(ref)) + 1e-30).all()
