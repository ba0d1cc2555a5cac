"""Cells with a plane test that FP32 leaves undecided have FP64 results in every form, the FP32 form included: a simple
cubic lattice with motion of 1e-6 of its spacing, where every cell has such tests, in sizes on either side of the lines
between the passes.  Against the FP64 oracle with the bar of the parity tests for such lattices (volumes 1e-11 relative;
areas by 1e-12 of their perimeter: the reference leaves a vertex where it is within 1e-12 of a plane)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("m", [5, 15, 17, 20, 21, 27])
def test_lattice_in_fp64(tess, oracle_mod, m, prec):
    g = np.arange(m) + 0.5
    pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    pts = (pts + 1e-6 * (np.random.default_rng(m).random(pts.shape) - 0.5)) / m
    r = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1])
    rv, ro, ri, ra, _, _ = r.compute_all()
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        d.compute_all(prec)
        vol = d.volumes()
        offs, nbr, area = d.neighbors_csr()
        assert d.stats()["rerun_fp64"] == len(pts)
    assert np.max(np.abs(vol - rv) / rv) <= 1e-11
    # faces larger than the motion makes: their neighbours and areas (slivers depend on the order of the cuts)
    big, rbig = area > 0.1 / m ** 2, ra > 0.1 / m ** 2
    assert np.array_equal(nbr[big], ri[rbig])
    assert np.max(np.abs(area[big] - ra[rbig])) <= 4e-12 / m
