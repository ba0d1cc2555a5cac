"""Where nearly every plane test is undecided (exact lattices) or points nearly coincide, cells go to the FP64 clipping and
are not settled test by test: by the passes' counters, in sizes on either side of the lines between the passes.  Volumes
against the exact ones of a lattice (1e-11 relative, the parity tests' bar) and the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def compute(tess, pts, prec):
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        d.compute_all(prec)
        return d.volumes(), d.neighbors_csr(), d.stats()


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("m", [10, 17, 21, 27, 33])
def test_exact_lattice(tess, m, prec):
    g = np.arange(m) + 0.5
    pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3) / m
    vol, _, st = compute(tess, pts, prec)
    assert np.max(np.abs(vol * m ** 3 - 1)) <= 1e-11
    assert st["rerun_fp64"] == len(pts) and st["rerun_fp64_full"] >= 0.9 * len(pts)


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [1000, 20000])
def test_near_coincident_pairs(tess, oracle_mod, n, prec):
    rng = np.random.default_rng(n)
    p = rng.random((n // 2, 3))
    pts = np.clip(np.concatenate([p, p + 1e-7 * (rng.random(p.shape) - 0.5)]), 0, 1)
    rv = oracle_mod.Diagram(pts, lo=[0, 0, 0], hi=[1, 1, 1]).compute_all()[0]
    vol, _, st = compute(tess, pts, prec)
    assert st["rerun_fp64"] == st["rerun_fp64_full"] == n
    assert np.max(np.abs(vol - rv) / rv) <= 1e-11
