"""Running peaks from whatever the caller's peak fields start at: a lowest value, a negative
zero, a value above every depth.

A peak raised from zero is the largest depth (speed) of the steps, neither ever being
negative; from any other start it must be the larger of the two.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STARTS = (-1.0, -9999.0, -np.inf, -0.0, 1e-3, 50.0)


def _peaks(precision, order, tile, start, lost=()):
    """Peaks and depth after nine steps of one storm; the peak fields start at `start` (None:
    the storm has none), the depths of the cells `lost` at NaN."""
    from his_gb300 import workloads as W
    from his_gb300.config import SolverConfig
    from his_gb300.engine import FloodEngine, Member
    storm = W.plain_small()
    m = Member(storm, torch.float64 if precision == "fp64" else torch.float32,
               torch.device("cuda", torch.cuda.current_device()), True, start is not None, {})
    wet = torch.rand(m.h.shape, generator=torch.Generator().manual_seed(3), dtype=torch.float64)
    m.h += (0.1 * (wet - 0.3).clamp(min=0.0)).to(m.h)
    for j in lost:
        m.h.view(-1)[j] = float("nan")
    if start is not None:
        start = torch.as_tensor(start).to(m.h).expand(m.h.shape)
        m.peak_h.copy_(start)
        m.peak_speed.copy_(start)
    fe = FloodEngine([m], SolverConfig(spatial_order=order, slot_width_frac=storm.slot_width_frac),
                     precision=precision, tile=tile, graph_steps=4)
    fe.advance(9)
    torch.cuda.synchronize()
    return (m.peak_h.cpu(), m.peak_speed.cpu(), m.h.cpu()) if start is not None else m.h.cpu()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("order,tile", [(2, (58, 16)), (1, (58, 16)), (2, (122, 48)), (2, (0, 0))])
def test_peaks_are_raised_from_any_start(precision, order, tile):
    zero_h, zero_s, h = _peaks(precision, order, tile, 0.0)
    assert float(zero_h.max()) > 1e-3 and float(zero_s.max()) > 1e-3 and bool((zero_h >= h).all())
    start = torch.tensor(STARTS, dtype=h.dtype)[torch.arange(h.numel()) % len(STARTS)].reshape(h.shape)
    got_h, got_s, got = _peaks(precision, order, tile, start)
    assert torch.equal(got, h) and torch.equal(_peaks(precision, order, tile, None), h)
    assert torch.equal(got_h, torch.maximum(start, zero_h))
    assert torch.equal(got_s, torch.maximum(start, zero_s))


@pytest.mark.parametrize("order,tile", [(2, (58, 16)), (1, (58, 16)), (2, (122, 48)), (2, (0, 0))])
def test_float32_peaks_rise_from_nan(order, tile):
    zero_h, zero_s, h = _peaks("fp32", order, tile, 0.0)
    got_h, got_s, got = _peaks("fp32", order, tile, float("nan"))
    assert torch.equal(got, h) and torch.equal(got_h, zero_h) and torch.equal(got_s, zero_s)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_lost_depth_raises_no_peak(precision):
    lost = (2500, 2501, 5000)
    got_h, _, got = _peaks(precision, 2, (58, 16), -2.0, lost)
    for j in lost:
        assert bool(got.view(-1)[j].isnan()) and float(got_h.view(-1)[j]) == -2.0
