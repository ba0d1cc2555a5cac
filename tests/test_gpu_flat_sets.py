"""Planes and lines of points, whose offsets of equal key are more than the shell table holds: whole diagrams, points
replaced, and single cells by index and by position, with a void that the walk crosses beyond the table.  Against the
FP64 oracle with the bars of the other tests (neighbour lists equal; volumes 1e-6 relative in FP32, 1e-12 otherwise;
1e-12 for vertices).  A line's cells are slices of the box between two cross-sections of area 1, as thin as 1e-5: in
FP64 each section's place is off by up to 2^-52, so their volumes have 2^-51 added to the bar (compared with exact
volumes, the oracle is off by 5e-17, which is 5e-12 of the thinnest)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def flat(n, axes, seed):
    """n points in the unit box at 0.25 on `axes`, none within 0.3 of the middle along the others."""
    rng = np.random.default_rng(seed)
    p = rng.random((4 * n, 3))
    p[:, list(axes)] = 0.25
    free = [a for a in range(3) if a not in axes]
    return np.ascontiguousarray(p[np.linalg.norm(p[:, free] - 0.5, axis=1) > 0.3][:n])


SETS = {"plane_x": (0,), "plane_y": (1,), "plane_z": (2,), "line_x": (1, 2), "line_z": (0, 1)}
BOX = (0, 0, 0, 1, 1, 1)


def sections(pts):
    return 2.0 ** -51 if np.sum(np.ptp(pts, axis=0) > 0) == 1 else 0.0


def check_all(d, oracle_mod, pts, prec):
    rv, ro, ri, _, _, _ = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).compute_all()
    d.compute_all(prec)
    vol = d.volumes()
    offs, nbr, _ = d.neighbors_csr()
    assert np.array_equal(offs.astype(np.int64), ro) and np.array_equal(nbr.astype(np.int64), ri)
    assert np.all(np.abs(vol - rv) <= (1e-6 if prec == "fp32" else 1e-12) * rv + sections(pts))


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [640, 915, 1300, 3000])
@pytest.mark.parametrize("name", list(SETS))
def test_whole_diagrams(tess, oracle_mod, name, n, prec):
    pts = flat(n, SETS[name], n)
    with tess.Diagram(pts, container=tess.Polyhedron(*BOX)) as d:
        check_all(d, oracle_mod, pts, prec)
        assert 1 <= d.stats()["table_entries"] <= 4096


@pytest.mark.parametrize("name", ["plane_z", "line_x"])
def test_points_replaced(tess, oracle_mod, name):
    """From a plane to points all over the box and back."""
    pts = flat(1500, SETS[name], 1)
    other = np.random.default_rng(2).random((1500, 3))
    with tess.Diagram(other, container=tess.Polyhedron(*BOX)) as d:
        for p in (pts, other, pts):
            d.update_points(p)
            check_all(d, oracle_mod, p, "fp64")


@pytest.mark.parametrize("n", [1300, 3000])
@pytest.mark.parametrize("name", list(SETS))
def test_single_cells(tess, oracle_mod, name, n):
    """Cells of the points around the void, and of positions in it: on the set, beside it, above and below."""
    pts = flat(n, SETS[name], n)
    axes = SETS[name]
    free = [a for a in range(3) if a not in axes]
    r = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1])
    rim = np.argsort(np.linalg.norm(pts[:, free] - 0.5, axis=1))[:6]
    where = []
    for h in (0.25, 0.25 + 1e-3, 0.25 - 1e-3, 0.2, 0.3):
        p = [0.5, 0.5, 0.5]
        for a in axes:
            p[a] = h
        where.append(p)
    with tess.Diagram(pts, container=tess.Polyhedron(*BOX)) as d:
        cells = [(d.get_cell_at_index(int(i)), r.cell(int(i))) for i in rim]
        cells += [(d.get_cell_at_particle(p), r.cell_at(p)) for p in where]
        for cell, ref in cells:
            if len(ref.vertices) > 255:
                with pytest.raises(tess.TessError, match="TESS_E_OVERFLOW"):
                    cell.compute_voronoi_cell()
                continue
            cell.compute_voronoi_cell()
            assert cell.compute_neighbors() == ref.ids.tolist()
            assert math.isclose(cell.compute_volume(), ref.volume, rel_tol=1e-12, abs_tol=sections(pts))
            v = np.asarray(cell.compute_vertices())
            dist = np.linalg.norm(v[:, None] - ref.vertices[None], axis=2)
            assert dist.min(axis=0).max() <= 1e-12 and dist.min(axis=1).max() <= 1e-12


def test_identical_points_seen_from_outside(tess, oracle_mod):
    """No axis has an extent: positions on either side of the one place that all points share."""
    pts = np.full((4, 3), 0.5)
    r = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1])
    with tess.Diagram(pts, container=tess.Polyhedron(*BOX)) as d:
        for p in ([0.4, 0.45, 0.3], [0.6, 0.55, 0.7], [0.4, 0.6, 0.5]):
            cell, ref = d.get_cell_at_particle(p).compute_voronoi_cell(), r.cell_at(p)
            assert cell.compute_neighbors() == ref.ids.tolist()
            assert math.isclose(cell.compute_volume(), ref.volume, rel_tol=1e-12)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_keys_that_underflow(tess, oracle_mod, prec):
    """Sides of 1e-171: every key is 0, and no whole key fits the table.  The oracle's cells (nothing cuts within the
    reference's tolerance)."""
    pts = np.random.default_rng(5).random((1300, 3)) * 1e-170
    box = [1e-170] * 3
    ro, ri = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=box).compute_all()[1:3]
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, *box)) as d:
        d.compute_all(prec)
        offs, nbr, _ = d.neighbors_csr()
        assert d.stats()["table_entries"] == 1
    assert np.array_equal(offs.astype(np.int64), ro) and np.array_equal(nbr.astype(np.int64), ri)
