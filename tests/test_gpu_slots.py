"""Without capacity re-runs, slots_per_lane says how large a cell may become: 64, 128 or 255 vertices with 2, 4 or 8.  A
site inside 45 or 90 points of a sphere has 86 or 176 vertices (2 f - 4 of f faces) that no other point cuts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(faces, n):
    """The site, its neighbours nearly on a sphere, and points away from it."""
    i = np.arange(faces) + 0.5
    z, a = 1 - 2 * i / faces, np.pi * (1 + 5 ** 0.5) * i
    u = np.stack([np.sqrt(1 - z * z) * np.cos(a), np.sqrt(1 - z * z) * np.sin(a), z], axis=1)
    rng = np.random.default_rng(faces)
    far = rng.random((4 * n, 3))
    far = far[np.linalg.norm(far - 0.5, axis=1) > 0.45][:n]
    return np.concatenate([[[0.5, 0.5, 0.5]], 0.5 + 0.1 * (1 + 1e-3 * rng.random((faces, 1))) * u, far])


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [200, 12000])
@pytest.mark.parametrize("faces,slots,fits", [(45, 2, False), (45, 4, True), (45, 8, True), (90, 2, False), (90, 4, False),
                                              (90, 8, True)])
def test_largest_cell(tess, oracle_mod, faces, slots, fits, n, prec):
    pts = points(faces, n)
    ref = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).cell(0)
    assert len(ref.vertices) == 2 * faces - 4
    cfg = tess.default_config(flags=tess.FLAG_NO_CAPACITY_RERUN, slots_per_lane=slots)
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1), config=cfg) as d:
        try:
            d.compute_all(prec)
        except tess.TessError as e:
            assert e.status == tess._capi.TESS_E_OVERFLOW
        nbr, _ = d.cell_faces(0)
        assert nbr.tolist() == (ref.ids.tolist() if fits else [])
