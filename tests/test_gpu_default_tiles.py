"""Decompositions left to the library, which choose them by the whole set.

A float32 member's totals are summed in float32 within a strip-chunk, so their last digits
follow the decomposition.  The server, whose results must not depend on who shares the
GPU, therefore fixes one.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_server_left_the_tile_uses_one_for_every_batch():
    from his_gb300 import workloads as W
    from his_gb300.engine import FloodEngine
    from his_gb300.serving import FloodServer
    storms = [W.uneven_member(f"serve-default/{k}", 0, 900.0 + 180.0 * k) for k in range(4)]
    srv = FloodServer(precision="fp32", chunk_steps=24, tile=(0, 0), keep_state=True)
    st = srv.serve([(0.0, s) for s in storms], max_wall_s=600)
    assert st.finished == 4 and st.max_members == 4
    by_key = {r.storm.key: r for r in srv.done}
    for s in storms:
        fe = FloodEngine([s], precision="fp32", tile=(58, 48), track_peaks=True)
        fe.run(chunk=128)
        assert np.array_equal(by_key[s.key].h, fe.h[0].cpu().numpy())
        assert by_key[s.key].result.sources == fe.results()[0].sources, s.key


# Relative bounds of a total between two decompositions: all its terms are >= 0, so a float32
# sum within a chunk, of up to 64 rows in a row and a tree of 6 levels over 64 columns, is off
# by at most 70 roundings of 2^-24, and two sums by twice that; float64 sums of the 8100
# cells by at most 2 x 8100 of 2^-53.
@pytest.mark.parametrize("dtype,rel", [(torch.float32, 140 * 2.0 ** -24), (torch.float64, 16200 * 2.0 ** -53)])
def test_a_member_alone_and_in_batches_left_the_tile(dtype, rel):
    from his_gb300.boundaries import EdgeBC
    from his_gb300.config import SolverConfig
    from his_gb300.infiltration import Horton
    from his_gb300.swe2d import SWE2D
    ny, nx = 81, 100
    y, x = np.mgrid[0:ny, 0:nx]
    z = 0.003 * x + 0.3 * np.sin(y / 7.0) * np.cos(x / 9.0)
    rng = np.random.default_rng(4)
    h0 = np.clip(0.4 + 0.1 * rng.random((ny, nx)) - z, 0.0, None)
    f0 = 1e-5 + 1e-5 * rng.random((ny, nx))
    bcs = {"west": EdgeBC("discharge", 0.3), "east": EdgeBC("stage", 0.35), "south": EdgeBC("transmissive"),
           "north": EdgeBC("closed")}

    def stepped(n):
        stack = lambda a: np.broadcast_to(a, (n, ny, nx)).copy()
        sim = SWE2D(z, 0.04, 10.0, SolverConfig(), bcs, dtype=dtype, batch=n,
                    horton=Horton(stack(f0), stack(0.1 * f0), stack(np.full((ny, nx), 1e-3))),
                    rain_weight=0.5 + x / nx)
        sim.set_state(*(torch.as_tensor(stack(a)) for a in (h0, 0.03 * h0, -0.02 * h0)))
        vols, dts = [], []
        for k in range(4):
            dts.append(sim.max_dt())
            vols.append(sim.step(dts[-1], 0.3 * k, 2e-5).table.cpu().numpy())
        return [getattr(sim, f)[0].cpu() for f in ("h", "hu", "hv", "infil_cum")], np.stack(vols, 1), dts

    state, alone, dts = stepped(1)
    assert alone[0, :, :4].min() > 0.0
    for n in (4, 16, 64):
        s, vols, d = stepped(n)
        assert d == dts and all(torch.equal(a, b) for a, b in zip(s, state)), n
        assert np.array_equal(vols, np.broadcast_to(vols[:1], vols.shape)), n
        assert (np.abs(vols[0] - alone[0]) <= rel * alone[0]).all(), n
