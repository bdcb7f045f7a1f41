"""Grids of one column or one row with open edges on both of its sides: how many segments a
strip-chunk is marched in does not change a bit of a member's state or totals."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ny,nx,tile", [(96, 1, (58, 48)), (90, 1, (58, 16)), (1, 200, (58, 16)), (2, 200, (58, 2)),
                                        (97, 2, (58, 48)), (90, 2, (1, 16))])
def test_segments_do_not_change_narrow_grids(ny, nx, tile, order):
    from his_gb300.boundaries import EdgeBC
    from his_gb300.config import SolverConfig
    from his_gb300.swe2d import SWE2D
    rng = np.random.default_rng(ny + nx)
    z = 0.3 * rng.random((ny, nx))
    h0, u, v = 0.5 + 0.2 * rng.random((ny, nx)), rng.normal(size=(ny, nx)), rng.normal(size=(ny, nx))
    bcs = {"west": EdgeBC("transmissive"), "east": EdgeBC("stage", 0.4), "south": EdgeBC("transmissive"),
           "north": EdgeBC("discharge", 0.2)}

    def stepped(n):
        stack = lambda a: np.broadcast_to(a, (n, ny, nx)).copy()
        sim = SWE2D(z, 0.03, 10.0, SolverConfig(spatial_order=order), bcs, dtype=torch.float32, batch=n, tile=tile)
        sim.set_state(*(torch.as_tensor(stack(a)) for a in (h0, h0 * u, h0 * v)))
        vols = [sim.step(0.2, 0.2 * k, 1e-5).table.cpu().numpy() for k in range(5)]
        return [getattr(sim, f)[0].cpu() for f in ("h", "hu", "hv")], np.stack(vols, 1)

    state, alone = stepped(1)                        # four segments where the chunk is tall enough
    assert alone[0, :, :2].min() > 0.0
    for n in (150, 1200):                            # two, one
        s, vols = stepped(n)
        assert all(torch.equal(a, b) for a, b in zip(s, state)), n
        assert np.array_equal(vols, np.broadcast_to(alone, vols.shape)), n
