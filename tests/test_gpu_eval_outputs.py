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
