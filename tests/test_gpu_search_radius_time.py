"""A search radius bounds the walk: cells that it leaves open (they reach far beyond the bins searched) take no longer than
closed ones.  The bar is loose, three times the time without a radius (walking every ring within reach took five times it
and more)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [3000, 50_000])
@pytest.mark.parametrize("radius", [0.0, 1e-4])
def test_open_cells(tess, radius, n, prec):
    pts = np.random.default_rng(n).random((n, 3))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        def once(r):
            t = time.perf_counter()
            d.compute_all(prec, search_radius=r)
            return time.perf_counter() - t
        for _ in range(3):
            once(None), once(radius)
        closed, open_ = (np.median([once(r) for _ in range(15)]) for r in (None, radius))
    assert open_ <= 3.0 * closed
