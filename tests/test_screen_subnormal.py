"""Double joins whose squared distances are subnormal in float.

Double data is screened in float before a distance is taken in double.  Below a
squared distance of about 1e-38 every multiply-add of the float chain rounds to
a multiple of 2^-149 instead of 24 bits, so a relative allowance does not cover
it: the screen's bound needs half such a step per dimension as well, or points
(and whole boxes) at the threshold distance are lost.

The sets make that matter.  Corners: a point and sign vectors around it, all at
one distance up to the last bit, so that the row is decided by the ids and a
candidate that the screen drops is missing from it.  Cloud: random points, and
the same beside points near 1, where the coordinates' size does not hide the
missing step.
"""
import numpy as np
import pytest

import oracle
import hybrid_k_nearest_neighbor_self_join_gb300 as kj

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()
    __graft_entry__.build_oracle()


def check(x, k, queries, di=0):
    ids, dists = kj.selfjoin(x, k, num_indexed_dims=di)
    perm, _ = kj.reorder_dims(x)
    bi, bd = oracle.bruteforce(np.ascontiguousarray(x[:, perm]), k + 1, queries.astype(np.uint32))
    assert np.array_equal(ids[queries], bi)
    assert np.array_equal(dists[queries].view(np.uint64), bd.view(np.uint64))


# offsets whose squares round up in float (in 12, 16 and 40 equal terms the chain
# ends above a bound without the absolute term)
SIZES = [2.7e-23, 1.7e-22, 4.5e-22, 1.2e-21, 3.6e-21]


@pytest.mark.parametrize("d", [12, 16, 40])
def test_corners(d):
    rng = np.random.default_rng(d)
    for c in SIZES:
        x = c * rng.choice([-1.0, 1.0], (3000, d))
        centre = rng.integers(0, 3000, 24)
        x[centre] = 0.0
        check(x, 40, centre)


@pytest.mark.parametrize("d", [12, 40, 128])
@pytest.mark.parametrize("beside", [False, True])
def test_cloud(d, beside):
    rng = np.random.default_rng(100 + d)
    for c in SIZES:
        x = rng.uniform(-c, c, (1500, d))
        if beside:
            x = np.concatenate([x, rng.uniform(0.5, 1.0, (1500, d))])
        # (more indexed dimensions are refused beside points near 1: over 2^64 cells)
        check(x, 24, np.arange(0, 1500, 7), di=2)


@pytest.mark.parametrize("d", [12, 40])
def test_corners_ring_search(monkeypatch, d):
    # the grid's ring search has a screen of its own
    monkeypatch.setenv("KNNSJ_TREE", "0")
    rng = np.random.default_rng(200 + d)
    for c in SIZES[1:4]:
        x = c * rng.choice([-1.0, 1.0], (700, d))
        centre = rng.integers(0, 700, 8)
        x[centre] = 0.0
        check(x, 20, centre)
