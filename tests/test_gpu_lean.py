"""The FP32 passes on the point sets where their walk over rows of bins can go wrong: axes without extent, oblong
grids, sparse regions that need rings of rows far out (more rows than lanes in a ring), sizes around a window of 32
candidates and around the size from which the plain, dense and careful passes share the work, lone points beside a cloud
of thousands (handed on for the length of their batches), extents outside FP32's
range, and a search radius, all against the FP64 oracle with the bars of the parity tests (neighbour lists bit-exact;
volumes 1e-6 relative in FP32, 1e-12 in MIXED and FP64)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOL_TOL = {"mixed": 1e-12, "fp64": 1e-12, "fp32": 1e-6}

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _rng(seed):
    return np.random.default_rng(seed)


def _clumps(n, clumps, seed, size=0.004, lone=40):
    """Points in tight clumps and a few lone ones between them: most bins are empty."""
    r = _rng(seed)
    c = 0.05 + 0.9 * r.random((clumps, 3))
    return np.concatenate([c[r.integers(0, clumps, n - lone)] + size * (r.random((n - lone, 3)) - 0.5), r.random((lone, 3))])


def _flat(pts, axis, value):
    pts[:, axis] = value
    return pts


def _clustered(n):
    from tessellator import workloads

    return workloads.clustered(n, seed=3)


SETS = {
    **{f"uniform_{n}": (lambda n=n: _rng(n).random((n, 3)), (1, 1, 1)) for n in (1, 2, 3, 31, 32, 33, 34, 64, 65, 200)},
    **{f"uniform_{n}": (lambda n=n: _rng(n).random((n, 3)), (1, 1, 1)) for n in (8192, 8193)},
    "clustered_40000": (lambda: _clustered(40_000), (1, 1, 1)),
    "plane_x": (lambda: _flat(_rng(1).random((300, 3)), 0, 0.25), (1, 1, 1)),
    "plane_y": (lambda: _flat(_rng(2).random((300, 3)), 1, 0.5), (1, 1, 1)),
    "plane_z": (lambda: _flat(_rng(3).random((300, 3)), 2, 0.75), (1, 1, 1)),
    "line": (lambda: _flat(_flat(_rng(4).random((60, 3)), 0, 0.5), 2, 0.5), (1, 1, 1)),
    "oblong_x": (lambda: _rng(5).random((3000, 3)) * [20, 1, 1], (20, 1, 1)),
    "oblong_y": (lambda: _rng(6).random((3000, 3)) * [1, 20, 0.5], (1, 20, 0.5)),
    "oblong_z": (lambda: _rng(7).random((3000, 3)) * [0.5, 1, 20], (0.5, 1, 20)),
    "clumps_few": (lambda: _clumps(1500, 4, 8), (1, 1, 1)),
    "clumps_many": (lambda: _clumps(20000, 60, 9), (1, 1, 1)),
    "beside_cloud": (lambda: _clumps(12000, 2, 12, size=0.15, lone=2000), (1, 1, 1)),
    "lone_corner": (lambda: np.concatenate([0.9 + 0.1 * _rng(10).random((4000, 3)), [[0.01, 0.02, 0.03]]]), (1, 1, 1)),
}


def _check(T, O, pts, hi, prec, ref_kw, **kw):
    rv, ro, ri, _, _, _ = O.Diagram(pts, lo=[0, 0, 0], hi=list(hi)).compute_all(**ref_kw)
    with T.Diagram(pts, container=T.Polyhedron(0, 0, 0, *hi)) as d:
        d.compute_all(prec, **kw)
        vol = d.volumes()
        offs, nbr, _ = d.neighbors_csr()
    assert np.array_equal(offs.astype(np.int64), ro)
    assert np.array_equal(nbr.astype(np.int64), ri)
    assert np.max(np.abs(vol - rv) / np.maximum(rv, 1e-300)) <= VOL_TOL[prec]


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("name", list(SETS))
def test_point_sets(tess, oracle_mod, name, prec):
    make, hi = SETS[name]
    _check(tess, oracle_mod, np.ascontiguousarray(make(), dtype=np.float64), hi, prec, {})


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("radius", [0.0, 0.01, 0.09, 0.5])
@pytest.mark.parametrize("name", ["uniform_200", "oblong_x", "clumps_few"])
def test_search_radius(tess, oracle_mod, name, radius, prec):
    make, hi = SETS[name]
    _check(tess, oracle_mod, np.ascontiguousarray(make(), dtype=np.float64), hi, prec,
           {"mode": oracle_mod.MODE_RADIUS, "radius": radius}, search_radius=radius)


def test_extent_below_fp32(tess, oracle_mod):
    """Bin sides below FP32's normal range: the pass hands every cell on."""
    _check(tess, oracle_mod, _rng(11).random((100, 3)) * 1e-42, (1e-42, 1e-42, 1e-42), "fp32", {})


def test_checked_build():
    """The plain, dense and careful passes through the bounds-checked library."""
    env = dict(os.environ, TESS_LIB=os.path.join(ROOT, "the-tessellator_gb300", "tessellator", "libtessgpu_checked.so"))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.abspath(__file__), "-q", "-x", "-m", "gpu", "-k",
                        "uniform_8193 or clustered_40000 or clumps_many"], env=env, cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "passed" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
