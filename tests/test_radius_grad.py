"""The training kernel's gradient at the edges of its tiles (64 samples) and of
its persistent grid (304 blocks: from 19 457 samples on blocks walk over several
tiles), against a numpy restatement in double."""
import ctypes

import numpy as np
import pytest

from hybrid_k_nearest_neighbor_self_join_gb300 import _lib
from test_learned_radius import NF, np_grad, random_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 19_456, 19_457, 45_001])
def test_gradient_at_tile_edges(n):
    m = random_model(11)
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, NF)).astype(np.float32)
    Y = rng.normal(0, 1, n).astype(np.float32)
    g = np.empty(_lib.RADIUS_MODEL_FLOATS - 2 * NF, np.float32)
    loss = ctypes.c_double(0)
    _lib.check(_lib.load().knnsj_radius_grad(m.ctypes.data, X.ctypes.data, Y.ctypes.data, n, 0.9, g.ctypes.data,
                                             ctypes.byref(loss)))
    want, wl = np_grad(m, X, Y, 0.9)
    # float sums of at most 64 * 3 + 38 + 8 terms per parameter: 238 * 2^-24
    # of the sum of magnitudes, which stays within a few times the largest
    # entry; activations carry 90 roundings
    assert np.max(np.abs(g - want)) <= 1e-4 * np.abs(want).max() + 1e-6
    assert abs(loss.value - wl) <= 1e-5 * abs(wl) + 1e-6
