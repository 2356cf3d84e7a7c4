"""A point's results do not depend on how many points share the call: with one
batched shape its tile sums are the same, and so must be what is made of them, to
the last bit.  The calls are on both sides of every limit of points where the
kernel cuts its work another way, over bins of one slot and of more than its runs."""
import numpy as np
import pytest

from gundam_gb300 import Engine
from gundam_gb300 import _native as N

pytestmark = pytest.mark.gpu

POINTS = (2, 3, 4, 5, 8, 9, 15, 16, 17, 32, 33, 63)
EVENTS = (1, 40, 256, 300, 900, 2100, 2400, 5000)  # per bin: a slot holds at most 256


def _engine(llh_type, n_bins=len(EVENTS)):
    rng = np.random.default_rng(8)
    bins = np.repeat(np.arange(len(EVENTS)), EVENTS)
    if n_bins > len(EVENTS):  # and many bins of a few events, none empty (a Poisson term without expectation is inf)
        bins = np.concatenate([bins, np.arange(len(EVENTS), n_bins), rng.integers(len(EVENTS), n_bins, 4 * n_bins)])
    e = Engine(bins.size, 16, n_bins, k_max=64, precision="fp64")
    e.set_event_indices(bins.astype(np.int32))
    e.set_initial_values(rng.uniform(0.5, 1.5, bins.size))
    one = np.arange(bins.size, dtype=np.int32)
    e.add_dials(np.full(bins.size, N.GW_DIAL_NORM, np.uint8), one, rng.integers(0, 16, bins.size).astype(np.int32),
                np.full(bins.size, -1, np.int32), np.zeros(bins.size + 1, np.int64), np.zeros(0))
    e.set_data(rng.poisson(np.bincount(bins, minlength=n_bins)).astype(np.float64))
    e.set_likelihood(llh_type)
    e.set_prior(np.ones(16), np.eye(16))
    e.initialize()
    return e, rng.uniform(0.7, 1.3, (64, 16))


def _batched_shapes(e):
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
    assert len(done) >= 3


def test_sums_of_a_point_at_every_number_of_points():
    e, pts = _engine(N.GW_LLH_NONE)
    for kind in _batched_shapes(e):
        sums, sums2, _, _ = e.eval(pts)
        for k in POINTS:
            s, s2, _, _ = e.eval(pts[:k])
            assert np.array_equal(s, sums[:k]) and np.array_equal(s2, sums2[:k]), (kind, k)
    e.close()


# bins: one part of 8, one group of 256 and a bin, more groups than runs, and so many
# that one point's parts are added in two levels as well
@pytest.mark.parametrize("n_bins", [8, 257, 2500, 17000])
@pytest.mark.parametrize("llh_type", [N.GW_LLH_POISSON, N.GW_LLH_BARLOW_BEESTON_OA2021])
def test_likelihood_of_a_point_at_every_number_of_points(llh_type, n_bins):
    torch = pytest.importorskip("torch")
    e, pts = _engine(llh_type, n_bins)
    rng = np.random.default_rng(8)
    data = rng.poisson(rng.uniform(0.0, 9.0, n_bins)).astype(np.float64)
    e.set_data(data)
    d_data = torch.from_numpy(data).cuda()
    for kind in _batched_shapes(e):
        _, _, llh, stat = e.eval(pts)
        for k in POINTS + (1, 64):
            s, s2, f, t = e.eval(pts[:k])
            assert np.isfinite(t).all()
            if k > 1:  # one point has kernels, and so tile sums, of its own
                assert np.array_equal(f, llh[:k]) and np.array_equal(t, stat[:k]), (kind, k)
            # the same from the sums
            d_s, d_s2 = torch.from_numpy(s).cuda(), torch.from_numpy(s2).cuda()
            out = torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert N.libgw().gw_llh_noalloc(d_s.data_ptr(), d_s2.data_ptr(), d_data.data_ptr(), n_bins, k, llh_type,
                                            out.data_ptr(), None) == N.GW_OK
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), t), (kind, k)
    e.close()
