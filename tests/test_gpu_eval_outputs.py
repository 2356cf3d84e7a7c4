"""gw_eval's outputs: what arrives in each array, for every choice of arrays and size
of the result."""
import numpy as np
import pytest

from gundam_gb300 import Engine, Workload
from gundam_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_without_a_likelihood_both_are_zero(graph):
    wl = Workload("mixed", seed=11)
    e = Engine.from_workload(wl, precision="fp64", k_max=8, llh_type=N.GW_LLH_NONE)
    e.use_graph(graph)
    for k in (8, 3, 1, 8):  # the results of one call lie where another's bin sums lay
        sums, _, llh, stat = e.eval(wl.draw_points(k, 2))
        assert sums.any()
        assert np.array_equal(llh, np.zeros(k)) and np.array_equal(stat, np.zeros(k))
    e.close()


@pytest.mark.parametrize("graph", [False, True])
def test_every_choice_of_arrays_small_and_large(graph):
    """The block of results travels as far as the last array asked for, in one copy
    or, from 4 MB on, in four: 9000 bins are below that with 3 points, above it with
    64, and with 40 above it only with both sums."""
    torch = pytest.importorskip("torch")
    n_bins, n = 9000, 20000
    rng = np.random.default_rng(6)
    e = Engine(n, 8, n_bins, k_max=64, precision="fp64")
    e.set_event_indices(np.concatenate([np.arange(n_bins), rng.integers(0, n_bins, n - n_bins)]).astype(np.int32))
    e.set_initial_values(rng.uniform(0.5, 1.5, n))
    e.add_dials(np.full(n, N.GW_DIAL_NORM, np.uint8), np.arange(n, dtype=np.int32),
                rng.integers(0, 8, n).astype(np.int32), np.full(n, -1, np.int32), np.zeros(n + 1, np.int64), np.zeros(0))
    e.set_data(rng.poisson(2.0, n_bins).astype(np.float64))
    e.set_likelihood(N.GW_LLH_BARLOW_BEESTON_OA2021)
    e.set_prior(np.ones(8), np.eye(8))
    e.initialize()
    e.use_graph(graph)
    lib = N.libgw()
    for rep, k in enumerate((3, 64, 40, 3)):
        pts = rng.uniform(0.5, 1.5, (k, 8))
        d_p = torch.from_numpy(pts).cuda()
        dev = [torch.empty(s, dtype=torch.float64, device="cuda") for s in (k * n_bins, k * n_bins, k, k)]
        torch.cuda.synchronize()
        e.eval_device(d_p.data_ptr(), k, *[t.data_ptr() for t in dev])
        e.sync()
        ref = [t.cpu().numpy() for t in dev]
        for want in range(16):
            out = [np.full(r.size, -1.0) if want >> i & 1 else None for i, r in enumerate(ref)]
            rc = lib.gw_eval(e._e, pts.ctypes.data, k, *[None if a is None else a.ctypes.data for a in out])
            assert rc == N.GW_OK
            for i, a in enumerate(out):
                assert a is None or np.array_equal(a, ref[i]), (rep, k, want, i)
    e.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64", "df64"])
def test_one_point_on_a_callers_stream(precision):
    """The one-point chain of dependent launches, direct and as a graph, replayed with
    other points in the same buffer."""
    torch = pytest.importorskip("torch")
    wl = Workload("mixed", seed=9)
    e = Engine.from_workload(wl, precision=precision, k_max=1, llh_type=N.GW_LLH_BARLOW_BEESTON_OA2021)
    pts = wl.draw_points(6, 4)
    ref = [e.eval(p[None]) for p in pts]
    stream = torch.cuda.Stream()
    d_p = torch.empty((1, wl.n_params), dtype=torch.float64, device="cuda")
    dev = [torch.empty(s, dtype=torch.float64, device="cuda") for s in (wl.n_bins, wl.n_bins, 1, 1)]
    for graph in (False, True, False):
        e.use_graph(graph)
        for p, r in zip(pts, ref):
            d_p.copy_(torch.from_numpy(p[None]))
            torch.cuda.synchronize()
            for _ in range(2):  # back to back
                e.eval_device(d_p.data_ptr(), 1, *[t.data_ptr() for t in dev], stream.cuda_stream)
            stream.synchronize()
            e.sync()
            for t, want in zip(dev, r):
                assert np.array_equal(t.cpu().numpy(), want.ravel())
    e.close()
