"""Neighbours within a radius on either side of the sizes from which a lane answers a query instead of a warp: evenly filled
and crowded grids, by distance and by bins, against the oracle's lists (whole numbers, so equal)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(crowd):
    rng = np.random.default_rng(3)
    p = rng.random((4000, 3))
    if crowd:                  # a tenth in 20 clusters of several hundred times the density
        c = rng.random((20, 3))
        p[:400] = np.clip(c[rng.integers(0, 20, 400)] + 2e-3 * rng.standard_normal((400, 3)), 0, 1)
    return p


@pytest.mark.parametrize("crowd,real,nq", [(False, False, 16383), (False, False, 16384), (False, True, 16384), (True, False, 16384),
                                           (True, True, 8192), (True, True, 262143), (True, True, 262144)])
def test_lists(tess, oracle_mod, crowd, real, nq):
    pts = points(crowd)
    rng = np.random.default_rng(nq)
    q = -0.1 + 1.2 * rng.random((nq, 3))
    q[::3] = pts[rng.integers(0, len(pts), len(q[::3]))]
    with tess.Diagram(pts) as d:
        got = d.find_neighbors_in_radius_batch(q, 0.03, real)
    want = oracle_mod.Diagram(pts).find_neighbors_in_radius(q, 0.03, real)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


def test_crowd_follows_the_points(tess, oracle_mod):
    """Points replaced by crowded ones and back: the route is that of the present points."""
    rng = np.random.default_rng(9)
    q = rng.random((20_000, 3))
    with tess.Diagram(points(False)) as d:
        for crowd in (False, True, False):
            d.update_points(points(crowd))
            got = d.find_neighbors_in_radius_batch(q, 0.03, True)
            want = oracle_mod.Diagram(points(crowd)).find_neighbors_in_radius(q, 0.03, True)
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(got[1], want[1])
