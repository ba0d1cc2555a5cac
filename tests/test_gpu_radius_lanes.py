"""Neighbours within a radius with one query per lane (large batches), against
the oracle's lists: whole numbers, so equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LANES = 8192         # queries from which a lane answers one


def points(name):
    rng = np.random.default_rng(5)
    if name == "clumps":                     # rows of hundreds of points beside empty ones
        c = rng.random((6, 3))
        return np.concatenate([rng.random((2000, 3)), (c[:, None] + 2e-3 * rng.random((6, 700, 3))).reshape(-1, 3)])
    if name == "plane":
        p = rng.random((3000, 3))
        p[:, 1] = -0.5
        return p
    if name == "lattice":                    # distances equal to the radius
        g = np.arange(12.0)
        return np.stack(np.meshgrid(g, g, g), axis=-1).reshape(-1, 3)
    if name == "far":                        # large coordinates, small extent
        return 1e7 + rng.random((3000, 3))
    return rng.random((3000, 3)) * [4.0, 1.0, 0.01]


@pytest.mark.parametrize("name,radius", [("oblong", 0.05), ("oblong", 0.3), ("oblong", 0.0), ("clumps", 0.03), ("clumps", 0.001),
                                         ("plane", 0.08), ("lattice", 1.0), ("lattice", 2.0), ("far", 0.1)])
@pytest.mark.parametrize("nq", [LANES - 1, LANES, LANES + 33])
@pytest.mark.parametrize("real", [True, False])
def test_lists(tess, oracle_mod, name, radius, nq, real):
    pts = points(name)
    rng = np.random.default_rng(6)
    lo, hi = pts.min(axis=0), pts.max(axis=0)
    ext = np.maximum(hi - lo, 0.1)
    q = lo - 0.2 * ext + 1.4 * ext * rng.random((nq, 3))        # some off the grid
    q[::3] = pts[rng.integers(0, len(pts), len(q[::3]))]        # and some on a point
    q[1::97] += 1e4 * ext
    with tess.Diagram(pts) as d:
        got = d.find_neighbors_in_radius_batch(q, radius, real)
    want = oracle_mod.Diagram(pts).find_neighbors_in_radius(q, radius, real)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
