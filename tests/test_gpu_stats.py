"""tess_diagram_stats reports the last compute from the host: it neither waits for the handle's stream nor breaks a capture
that the caller runs on it, and points replaced since do not show."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_while_the_stream_is_captured(tess):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    pts = np.random.default_rng(1).random((3000, 3))
    with tess.Diagram(pts, container=tess.Polyhedron(0, 0, 0, 1, 1, 1),
                      config=tess.default_config(stream=stream.cuda_stream)) as d:
        d.compute_all("fp32")
        before = d.stats()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            x.add_(1.0)
            during = d.stats()
        graph.replay()
        torch.cuda.synchronize()
        assert during == before and before["table_entries"] > 1
        assert float(x[0]) == 1.0


def test_of_the_last_compute(tess):
    rng = np.random.default_rng(2)
    with tess.Diagram(rng.random((3000, 3)), container=tess.Polyhedron(0, 0, 0, 1, 1, 1)) as d:
        assert d.stats()["table_entries"] == 0
        d.compute_all("fp32")
        entries = d.stats()["table_entries"]
        d.update_points(rng.random((3000, 3)) * [1.0, 0.5, 0.01])
        assert d.stats()["table_entries"] == entries
        d.compute_all("fp32")
        assert 1 <= d.stats()["table_entries"] != entries
