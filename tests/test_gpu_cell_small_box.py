"""Single cells of boxes so small that the reference's tolerance (1e-12) takes faces away: a query in the FP32 form has
the faces of a whole compute in that form, which tests without the tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [1e-8, 1e-7, 1.0])
@pytest.mark.parametrize("n", [300, 9000])
def test_faces_of_the_whole_compute(tess, side, n):
    pts = np.random.default_rng(n).random((n, 3)) * side
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, side, side, side)) as d:
        d.compute_all("fp32")
        offs, nbr, _ = d.neighbors_csr()
        offs = offs.astype(np.int64)
        for i in range(0, n, max(1, n // 300)):
            want = nbr[offs[i]:offs[i + 1]].tolist()
            assert d.get_cell_at_index(i, precision="fp32").compute_voronoi_cell().compute_neighbors() == want
            if i % 7 == 0:
                corners = sum(len(d.cell_face_vertices(i, f)) for f in range(len(want)))
                assert corners == 3 * len(d.cell_vertices(i))
