"""eps_final of a join searched through the box tree is the largest radius it
searched: what was assigned, what a failed query grew to, or, without a radius,
the distance of the last neighbour."""
import math

import numpy as np
import pytest

import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import datasets, train_radius

pytestmark = pytest.mark.gpu

MARGIN = 0.08  # added to a predicted log radius (LEARNED_LOG_MARGIN)


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


@pytest.fixture
def constant_model():
    """A radius model that predicts log(radius / eps0) = y for every query."""
    def set_y(y):
        m = train_radius.placeholder_model()
        m[-1] = y
        kj.set_radius_model(m)
    yield set_y
    kj.set_radius_model(None)


@pytest.mark.parametrize("n,d,dtype", [(20_001, 4, np.float32), (10_000, 6, np.float64), (33, 4, np.float32)])
def test_learned_join(constant_model, n, d, dtype):
    x = datasets.gmm(n, d, 9, 0.2, 400 + d, dtype=dtype)
    k = 12
    dists, st0 = kj.selfjoin(x, k, return_stats=True)[1:]
    last = float(dists[:, k].max())
    # every query is found at the radius it is given: a half more than the
    # widest row needs
    y = math.log(1.5 * last / st0["eps0"])
    assert math.log(1.0 / 16.0) < y < math.log(60.0)
    constant_model(y)
    st = kj.selfjoin(x, k, radius_mode=kj.RADIUS_LEARNED, return_stats=True)[2]
    assert st["queries_run"] == n
    want = st["eps0"] * math.exp(y + MARGIN)
    # (the model's sums and exp in float)
    assert abs(st["eps_final"] - want) <= 1e-5 * want
    # and some are not: a tenth of that
    constant_model(y - math.log(10.0))
    st = kj.selfjoin(x, k, radius_mode=kj.RADIUS_LEARNED, return_stats=True)[2]
    assert st["queries_run"] > n
    assert st["eps_final"] >= last


@pytest.mark.parametrize("d,dtype", [(3, np.float32), (5, np.float64)])
def test_uniform_radius_join(d, dtype):
    x = datasets.gmm(20_003, d, 9, 0.2, 500 + d, dtype=dtype)
    k = 12
    ids, dists, st = kj.selfjoin(x, k, return_stats=True)
    assert st["eps_final"] >= max(st["eps0"], float(dists[:, k].max()))
