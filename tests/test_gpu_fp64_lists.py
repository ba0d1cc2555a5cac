"""The FP64 clipping at 64, 128 and 255 vertices: lists of cells shorter and longer than what decides between the first two,
in inputs on either side of the size from which there is a choice, with cells that outgrow each.  Near-coincident pairs
make the list, sites inside points of a sphere (with a near twin of their own) the large cells.  Against the FP64 oracle:
neighbour lists equal, the volumes of those cells 1e-11 relative (the parity tests' bar for such pairs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(n, npairs, seed):
    rng = np.random.default_rng(seed)

    def twins(p):
        return p + 1e-6 * (rng.random(p.shape) - 0.5)

    parts, centres = [], [[0.2, 0.2, 0.2], [0.8, 0.2, 0.3], [0.3, 0.8, 0.7]]
    for c, faces in zip(centres, (30, 90, 180)):
        i = np.arange(faces) + 0.5
        z, a = 1 - 2 * i / faces, np.pi * (1 + 5 ** 0.5) * i
        u = np.stack([np.sqrt(1 - z * z) * np.cos(a), np.sqrt(1 - z * z) * np.sin(a), z], axis=1)
        site = np.array([c])
        parts += [site, twins(site), c + 0.05 * (1 + 1e-3 * rng.random((faces, 1))) * u]
    far = rng.random((2 * n, 3))
    far = far[np.min(np.linalg.norm(far[:, None] - np.array(centres)[None], axis=2), axis=1) > 0.25]
    far = far[:n - npairs]
    pts = np.concatenate(parts + [far, twins(far[:npairs])])
    return np.clip(pts, 0.0, 1.0), [0, 1, 32, 33, 124, 125]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,npairs", [(5000, 300), (20000, 3000), (40000, 300), (40000, 3000)])
def test_lists_and_large_cells(tess, oracle_mod, n, npairs, prec):
    pts, sites = points(n, npairs, n + npairs)
    rv, ro, ri, _, _, _ = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).compute_all()
    faces = np.diff(ro)[sites]
    assert faces[0] < 30 < 40 < faces[2] < 66 < faces[4] < 128      # 64, 128 and 255 vertices
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        d.compute_all(prec)
        vol = d.volumes()
        offs, nbr, _ = d.neighbors_csr()
        st = d.stats()
    assert st["failed"] == 0 and st["rerun_fp64_full"] >= 2 * npairs
    assert np.array_equal(offs.astype(np.int64), ro) and np.array_equal(nbr.astype(np.int64), ri)
    full = np.concatenate([sites, np.arange(len(pts) - npairs, len(pts))])
    assert np.max(np.abs(vol[full] - rv[full]) / rv[full]) <= 1e-11
