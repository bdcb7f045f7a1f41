"""Infiltration rates below zero, the form of a spring: water they put on a dry cell comes
without momentum (the share of the momentum kept, new depth over old, is zero for a depth
of zero: swe2d.py:343-360)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ny,nx", [(30, 41), (205, 210)])          # float64: fused, faces apart
def test_a_spring_wets_dry_cells_without_momentum(dtype, order, ny, nx):
    from his_gb300.boundaries import all_edges
    from his_gb300.config import SolverConfig
    from his_gb300.infiltration import Horton
    from his_gb300.swe2d import SWE2D
    rate, dt = -2.0 ** -10, 4.0                      # 2^-8 m a step, exact in both precisions
    sim = SWE2D(torch.zeros(ny, nx, dtype=torch.float64), 0.03, 10.0, SolverConfig(spatial_order=order),
                all_edges("closed"), dtype=dtype,
                horton=Horton.constant(rate, (ny, nx), device="cuda", dtype=dtype))
    for k in (1, 2):
        sim.step(dt, dt * (k - 1))
        for name, want in (("h", k * -rate * dt), ("hu", 0.0), ("hv", 0.0), ("infil_cum", k * rate * dt)):
            assert torch.equal(getattr(sim, name), torch.full_like(sim.h, want)), (name, k)
