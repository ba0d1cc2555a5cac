"""The support tests that leave points of long batches out, checked on the CPU against exact arithmetic.

A bisector beyond the support of the box around a cell's vertices cuts nothing.  Both forms of that test are restated in
numpy float32 and held to the property the kernels rely on:

- FP64 clipping (csrc/tess_clip_impl.cuh, live_bounds): a candidate whose bisector has a vertex beyond it, by exact
  arithmetic on the FP64 positions, is kept, however near the vertex lies to the plane;
- FP32 passes (csrc/tess_clip_lean.cu, reaches): a candidate that touches a vertex by the FP32 plane test (beyond the
  plane or within the guard band) is kept.

Without their margins both lose such candidates, which shows that the samples come near enough to the boundary."""
from fractions import Fraction

import numpy as np
import pytest

F32 = np.float32
GUARD_REL, EC = F32(4e-7), F32(0.0)


def fma32(a, b, c):
    return F32(float(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c))))


def norm_up(x):
    """The kernel's upper bound of sqrt(x): within 2^-20 above the root."""
    return F32(np.sqrt(np.float64(x)) * (1.0 + 2.0 ** -21))


def exact_sd(r, v):
    r, v = [Fraction(float(x)) for x in r], [Fraction(float(x)) for x in v]
    return sum(a * b for a, b in zip(r, v)) - sum(a * a for a in r) / 2


def on_plane(rng, verts):
    """A candidate offset whose bisector passes through the vertex farthest along it: |r| = 2 max v.u."""
    u = rng.normal(size=3)
    u /= np.linalg.norm(u)
    return 2.0 * float(np.max(verts @ u)) * u


def box32(verts):
    """Bounds of the vertices' FP32 copies and the site, as the warp reduces them."""
    f = np.asarray(verts, dtype=np.float32)
    return np.minimum(f.min(axis=0), F32(0)), np.maximum(f.max(axis=0), F32(0))


def kept_fp64(r, verts, margin=True):
    r2 = float(r[0] * r[0] + r[1] * r[1] + r[2] * r[2])
    g, off = np.asarray(r, dtype=np.float32), F32(0.5) * F32(r2)
    lo, hi = box32(verts)
    h = F32(0)
    for a in range(3):
        h = F32(h + max(F32(g[a] * lo[a]), F32(g[a] * hi[a])))
    if not margin:
        return not h < off
    R = F32(np.sqrt(F32(max(float(v @ v) for v in verts))))
    slack = F32(F32(F32(4e-6) * F32(F32(abs(g[0]) + abs(g[1])) + abs(g[2]))) * R)
    return not F32(h * F32(1.000004) + slack) < F32(off * F32(0.999996))


@pytest.mark.parametrize("scale", [1.0, 1e-4, 1e5])
def test_fp64_clipping_keeps_every_cutter(scale):
    rng = np.random.default_rng(11)
    lost_without = cutters = 0
    for k in range(4000):
        # a cell as narrow as one vertex (the box touches it) up to one of a dozen
        verts = scale * rng.normal(size=(1 + k % 12, 3)) * 10.0 ** rng.uniform(-3, 0, size=3)
        r = on_plane(rng, verts) * (1.0 - 10.0 ** rng.uniform(-15, -6))
        if not r.any() or not any(exact_sd(r, v) > 0 for v in verts):
            continue
        cutters += 1
        assert kept_fp64(r, verts)
        lost_without += not kept_fp64(r, verts, margin=False)
    assert cutters > 1000 and lost_without > 10


def touched32(v, e, g, off, rn):
    sd = fma32(g[0], v[0], fma32(g[1], v[1], fma32(g[2], v[2], -off)))
    c0 = fma32(rn, fma32(GUARD_REL, rn, F32(0)), EC)
    return sd >= -fma32(rn, e, c0)


def kept_fp32(g, q2, n, verts, errs, margin=True):
    lo, hi = box32(verts)
    h = F32(F32(max(F32(g[0] * lo[0]), F32(g[0] * hi[0])) + max(F32(g[1] * lo[1]), F32(g[1] * hi[1]))) +
            max(F32(g[2] * lo[2]), F32(g[2] * hi[2])))
    if not margin:
        return h >= F32(0.5) * q2
    R2 = F32(max(float(norm_up(F32(v @ v)) + e) ** 2 for v, e in zip(verts, errs)))
    be = F32(max(errs) + F32(F32(1e-6) * norm_up(R2)))
    return F32(h + fma32(n, F32(be + fma32(GUARD_REL, n, F32(0))), EC)) >= F32(F32(0.5) * q2)


@pytest.mark.parametrize("scale", [1.0, 1e-4, 1e5])
def test_fp32_passes_keep_every_touched_candidate(scale):
    rng = np.random.default_rng(12)
    lost_without = hits = 0
    for k in range(4000):
        verts = (scale * rng.normal(size=(1 + k % 12, 3)) * 10.0 ** rng.uniform(-3, 0, size=3)).astype(np.float32)
        errs = (np.abs(verts).sum(axis=1) * 10.0 ** rng.uniform(-6.5, -3, size=len(verts))).astype(np.float32)
        g = (on_plane(rng, verts.astype(np.float64)) * (1.0 + rng.uniform(-1e-6, 2e-6))).astype(np.float32)
        q2 = F32(F32(F32(g[0] * g[0]) + F32(g[1] * g[1])) + F32(g[2] * g[2]))
        if not q2 > 0:
            continue
        n, off = norm_up(q2), F32(0.5) * q2
        if not any(touched32(v, e, g, off, n) for v, e in zip(verts, errs)):
            continue
        hits += 1
        assert kept_fp32(g, q2, n, verts, errs)
        lost_without += not kept_fp32(g, q2, n, verts, errs, margin=False)
    assert hits > 1000 and lost_without > 100
