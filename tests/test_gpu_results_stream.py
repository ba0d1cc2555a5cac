"""tess_results_device on the caller's own stream: volumes and offsets are complete on return, whatever else the GPU is
doing, and may be read on another stream (here by a copy engine, while every SM is busy with a third stream's work)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_offsets_complete_on_return(tess, batch):
    torch = pytest.importorskip("torch")
    n = 1_000_000
    gen = torch.Generator(device="cuda").manual_seed(3)
    first, second = (torch.rand(n, 3, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2))
    own, other, busy = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    work = torch.zeros(1 << 30, dtype=torch.float32, device="cuda")
    host = torch.empty(n + 1, dtype=torch.int64, pin_memory=True)
    torch.cuda.synchronize()
    cfg = tess.default_config(stream=own.cuda_stream)
    if batch:
        h = tess.Batch(first.cpu().numpy(), np.array([0, n // 2, n], dtype=np.uint64),
                       np.tile([0.0, 0.0, 0.0, 1.0, 1.0, 1.0], (2, 1)), config=cfg)
    else:
        h = tess.Diagram(container=tess.Polyhedron(0, 0, 0, 1, 1, 1), config=cfg, device_ptr=first.data_ptr(), n=n)
    try:
        for pts in (first, second):
            h.update_points(device_ptr=pts.data_ptr())
            h.compute("fp32") if batch else h.compute_all("fp32")
            with torch.cuda.stream(busy):
                for _ in range(8):
                    work.mul_(1.0)
            _, offs, _, _, total = h.results_device()
            view = torch.as_tensor(tess.DeviceArray(offs, n + 1, np.uint64), device="cuda").view(torch.int64)
            with torch.cuda.stream(other):
                host.copy_(view, non_blocking=True)
            other.synchronize()
            seen = host.numpy().copy()
            torch.cuda.synchronize()
            assert seen[n] == total
            assert np.array_equal(seen.astype(np.uint64), h.neighbors_csr()[0])
    finally:
        h.close()
