"""Cells of several hundred cuts through the FP32 passes, against the FP64 oracle: more planes than the plane table
holds (96), so that ids of faces cut away entirely are taken again, and more cuts than a ring map's tag counts (255), so
that the maps are cleared within a cell.  Shells of points around a site, the outermost stored first and no bin counted
as crowded: each window of candidates lies inside the one before it and cuts all its faces away."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shells(count, seed):
    """A site, `count` shells of 31 points inside one bin, outermost first, and points that span the box."""
    rng = np.random.default_rng(seed)
    u = rng.standard_normal((count, 31, 3))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    r = 0.05 * 0.9 ** np.arange(count)
    corners = np.array([[x, y, z] for x in (0.0, 1.0) for y in (0.0, 1.0) for z in (0.0, 1.0)])
    site = np.full(3, 0.93)            # (bins of a seventh to a tenth of the box: the middle of one)
    return np.concatenate([[site], (site + r[:, None, None] * u).reshape(-1, 3), corners, rng.random((40, 3))])


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("count", [4, 9, 20])
def test_planes_taken_again(tess, oracle_mod, count, prec):
    pts = shells(count, count)
    rv, ro, ri, _, _, _ = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).compute_all()
    cfg = tess.default_config(crowded_bin=1 << 20, flags=tess.FLAG_COUNTERS)
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1), config=cfg) as d:
        d.compute_all(prec)
        vol = d.volumes()
        offs, nbr, _ = d.neighbors_csr()
        stats = d.stats()
    print(count, prec, "cuts a cell", stats["cuts"] / len(pts), "re-run for capacity", stats["rerun_capacity"])
    assert np.array_equal(offs.astype(np.int64), ro) and np.array_equal(nbr.astype(np.int64), ri)
    assert np.max(np.abs(vol - rv) / rv) <= (1e-6 if prec == "fp32" else 1e-12)
