"""tess_stats.launches counts the kernels that a handle launches, on either side of the sizes at which a scan takes one
launch or three, queries are put in order, and lists overflow."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,crowd,want", [
    (1000, False, 1 + 1 + 1 + 1),            # count, scan, copy of the offsets, fill
    (16384, False, 1 + 1 + 1 + 1),
    (16385, False, 1 + 3 + 1 + 1),
    (262_144, True, 1 + 3 + 1 + 2),          # the listed results to their places, the others found again
    (600_000, False, 3 + 1 + 3 + 1 + 1),     # order: bins, scan, scatter
])
def test_radius_queries(tess, nq, crowd, want):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    pts = rng.random((20_000, 3))
    if crowd:
        pts[:2000] = 0.5 + 1e-3 * rng.random((2000, 3))
    q = torch.from_numpy(rng.random((nq, 3))).to("cuda")
    q[0] = 0.5005
    offs = torch.empty(nq + 1, dtype=torch.int64, device="cuda")
    ids = torch.empty(16 * nq + 4096, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        total = C.c_size_t(0)
        counts = []
        for _ in range(3):
            tess._capi.check(tess.lib().tess_find_neighbors_in_radius(
                d._h, q.data_ptr(), nq, 0.03, 1, 1, offs.data_ptr(), ids.data_ptr(), len(ids), C.byref(total)))
            counts.append(d.stats()["launches"])
    assert total.value > 0
    assert np.diff(counts).tolist() == [want, want]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [500, 9000])
def test_batch_and_diagram_count_alike(tess, prec, n):
    """The first compute of a batch, which captures its graph, and later ones; beside a diagram of the same points, which
    has no cell for the pass over the largest cells and leaves it out."""
    pts = np.random.default_rng(5).random((n, 3))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        start = d.stats()["launches"]
        d.rebuild()
        d.compute_all(prec)
        want = d.stats()["launches"] - start + 1
    b = tess.Batch(pts, np.array([0, n], dtype=np.uint64), np.array([[0.0, 0.0, 0.0, 1.0, 1.0, 1.0]]))
    try:
        start = b.stats()["launches"]
        for k in range(1, 4):
            b.compute(prec)
            assert b.stats()["launches"] - start == k * want
    finally:
        b.close()


def test_single_cell(tess):
    pts = np.random.default_rng(6).random((1000, 3))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        d.get_cell_at_index(3).compute_voronoi_cell()
        start = d.stats()["launches"]
        d.get_cell_at_index(4).compute_voronoi_cell()
        assert d.stats()["launches"] == start + 1


@pytest.mark.parametrize("p,launches", [((0.4, 0.5, 0.6), 1), ((0.4, 0.5, 1.6), 1), ((0.4, 0.5, 1.0), 1), ((-1e-9, 0.5, 0.6), 1)])
def test_cell_at_a_position(tess, oracle_mod, p, launches):
    """Inside the container, above it, on its wall, just below it: one launch each."""
    pts = np.random.default_rng(7).random((1000, 3))
    ref = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).cell_at(list(p))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        start = d.stats()["launches"]
        cell = d.get_cell_at_particle(list(p)).compute_voronoi_cell()
        assert d.stats()["launches"] == start + launches
        assert cell.compute_neighbors() == ref.ids.tolist()
