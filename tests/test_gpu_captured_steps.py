"""Steps in a graph of the caller's own, and what a handle that was captured leaves behind."""
import gc

import pytest
import torch

import test_gpu_graph_launches as G

pytestmark = pytest.mark.gpu


def test_a_captured_coupled_step_replays():
    a, b = G._coupled(1), G._coupled(1)
    dt, side = 0.25 * a.two.max_dt(), torch.cuda.Stream()
    la, lb = (torch.zeros((8, 1), dtype=torch.float64, device="cuda") for _ in range(2))
    rate = torch.zeros(2, dtype=torch.float64, device="cuda")
    for _ in range(2):                               # a plain call and the library's own graph
        G._in_one(a, a.one, dt, 0.0, la, rate, 2, side)
        G._separately(b, dt, 0.0, lb, 2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        G._in_one(a, a.one, dt, 0.0, la, rate, 2, side)
    for _ in range(3):
        g.replay()
        G._separately(b, dt, 0.0, lb, 2)
    G._same(a, b, a.one, la, lb, rate)
    # the slot the graph copies from is not given out again: that is an error of this call, and
    # neither it nor the handle's end is one of the caller's next
    refused = 0
    for _ in range(12):
        try:
            G._in_one(a, a.one, dt, 0.0, la, rate, 2, side)
        except RuntimeError:
            refused += 1
        assert float(torch.ones(4, device="cuda").sum()) == 4.0
    assert refused > 0
    # nor is it freed for larger ones: 256 substeps' forcing
    with pytest.raises(RuntimeError):
        G._in_one(a, a.one, dt, 0.0, la, rate, 256, side)
    assert float(torch.ones(4, device="cuda").sum()) == 4.0
    del a, g
    gc.collect()
    assert float(torch.ones(4, device="cuda").sum()) == 4.0
