"""The autotuner times what differs: knob sets that launch the same kernels are timed once, and no set but the default is
chosen for noise (compared by the handle's launch count, and by tuning the same input again and again)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PASSES = 5      # plain, dense, careful, FP64 clipping at 128 and 255 vertices
SETS = 4        # crowded-bin thresholds


def test_equal_launches_are_timed_once(tess):
    pts = np.random.default_rng(8).random((20_000, 3))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        for _ in range(6):
            start = d.stats()["launches"]
            t = d.autotune("fp32", cache_path="")
            assert t["trials"] == 2 * SETS
            assert d.stats()["launches"] - start == SETS * 2 * PASSES      # two runs each
            assert t["warps_per_block"] == 8                               # the default
