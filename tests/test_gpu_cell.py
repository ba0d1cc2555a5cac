"""One cell with its geometry (tess_cell_compute, tess_cell_compute_at) where
its kernel hands over to the FP64 form or the site and the container are not
the diagram's own, against the FP64 oracle.

Bars, as for the other FP64-finished cells of a unit box: the same neighbours,
volumes within 1e-12 relative, vertices within 1e-12, areas within 1e-10
relative.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(cell, ref):
    assert cell.compute_neighbors() == ref.ids.tolist()
    assert math.isclose(cell.compute_volume(), ref.volume, rel_tol=1e-12)
    v = np.asarray(cell.compute_vertices())
    assert len(v) == len(ref.vertices)
    d = np.linalg.norm(v[:, None] - ref.vertices[None], axis=2)
    assert d.min(axis=0).max() <= 1e-12 and d.min(axis=1).max() <= 1e-12
    for f, area, fv in zip(cell.compute_faces(), ref.areas, ref.face_vertices):
        assert math.isclose(f.compute_area(), area, rel_tol=1e-10, abs_tol=1e-15)
        got = np.asarray(f.compute_vertices())
        assert len(got) == len(fv)
        k = int(np.argmin(np.linalg.norm(got - fv[0], axis=1)))
        np.testing.assert_allclose(np.roll(got, -k, axis=0), fv, atol=1e-12)


def point_set(name):
    rng = np.random.default_rng(71)
    if name == "inner":                      # the grid covers a small part of the box
        return 0.4 + 0.2 * rng.random((800, 3))
    if name == "clump":                      # crowded bins: 300 of 900 points in 1e-3
        return np.concatenate([rng.random((600, 3)), 0.31 + 1e-3 * rng.random((300, 3))])
    if name == "plane":                      # an axis without extent
        p = rng.random((300, 3))
        p[:, 2] = 0.25
        return p
    assert name == "sphere"                  # point 0 has 120 faces
    u = rng.normal(size=(120, 3))
    return 0.5 + np.concatenate([np.zeros((1, 3)), 0.4 * u / np.linalg.norm(u, axis=1, keepdims=True)])


@pytest.mark.parametrize("name,index", [("inner", 3), ("clump", 5), ("clump", 700), ("plane", 8), ("sphere", 0),
                                        ("sphere", 60)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_cell_of_point(tess, oracle_mod, name, index, prec):
    pts = point_set(name)
    r = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1])
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        check(d.get_cell_at_index(index, precision=prec).compute_voronoi_cell(), r.cell(index))


@pytest.mark.parametrize("name", ["inner", "plane"])
@pytest.mark.parametrize("p", [(0.03, 0.9, 0.5), (0.999, 0.001, 0.002), (0.45, 0.52, 0.9), (0.45, 0.52, 0.1)])
def test_cell_at_any_point(tess, oracle_mod, name, p):
    """Sites off the grid of the points' bounds.  (Above the plane a cell has
    more vertices than a query returns, TESS_MAX_CELL_VERTICES.)"""
    pts = point_set(name)
    r = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1])
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        ref = r.cell_at(list(p))
        if len(ref.vertices) > 255:
            with pytest.raises(tess.TessError, match="TESS_E_OVERFLOW"):
                d.get_cell_at_particle(list(p)).compute_voronoi_cell()
        else:
            check(d.get_cell_at_particle(list(p)).compute_voronoi_cell(), ref)


@pytest.mark.parametrize("lo,hi", [((0.0, 0.0, 0.0), (1.0, 1.0, 1.0)), ((-3.0, -2.0, 0.39), (0.61, 5.0, 4.0))])
@pytest.mark.parametrize("radius,group", [(None, None), (0.01, None), (None, 1), (0.02, 1)])
def test_cell_with_container_radius_group(tess, oracle_mod, lo, hi, radius, group):
    pts = point_set("inner")
    groups = (np.arange(len(pts)) % 3).astype(np.uint32)
    r = oracle_mod.Diagram(pts, groups=groups, lo=list(lo), hi=list(hi))
    mode = oracle_mod.MODE_SECURE if radius is None else oracle_mod.MODE_RADIUS
    with tess.Diagram(pts, groups=groups, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        for i in (0, 411):
            cell = d.get_cell_at_index(i, polyhedron=tess.Polyhedron(*lo, *hi), search_radius=radius, target_group=group)
            check(cell.compute_voronoi_cell(), r.cell(i, mode=mode, radius=-1.0 if radius is None else radius,
                                                      target_group=-1 if group is None else group))
