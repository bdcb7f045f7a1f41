"""A float32 strip-chunk marched in one, two or four segments gives the same bits.

How many segments a set's chunks are marched in follows from how many chunks the set
has, so a member stepped alone (four segments), in a batch of 24 to 30 (two) and of 64
or more (one) takes different kernels.  States, volumes, rates and peaks must agree
exactly: a cell's arithmetic is the same in every march, and the rows' sums are added
in the same order.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FIELDS = ("h", "hu", "hv", "s_filled", "infil_cum")


def _sim(z, members, order, tile, rain_weight, sources):
    from his_gb300.boundaries import EdgeBC
    from his_gb300.config import SolverConfig
    from his_gb300.infiltration import Horton
    from his_gb300.swe2d import SWE2D
    ny, nx = z.shape
    B = len(members)
    rng = [np.random.default_rng(100 + m) for m in members]
    field = lambda lo, hi: np.stack([lo + (hi - lo) * g.random((ny, nx)) for g in rng])
    n = field(0.03, 0.05)
    kw = dict(storage=field(0.0, 0.002), horton=Horton(field(1e-5, 2e-5), field(1e-6, 2e-6), field(1e-3, 2e-3), 5.0)) \
        if sources else {}
    if rain_weight:
        kw["rain_weight"] = 0.5 + np.random.default_rng(1).random((ny, nx))
    bcs = {"west": EdgeBC("discharge", 0.3), "east": EdgeBC("stage", 0.35), "south": EdgeBC("transmissive"),
           "north": EdgeBC("closed")}
    sim = SWE2D(z, n, 10.0, SolverConfig(spatial_order=order), bcs, dtype=torch.float32, batch=B, tile=tile, **kw)
    h0 = np.clip(0.4 + field(0.0, 0.1) - z[None], 0.0, None)
    sim.set_state(h0, 0.03 * h0, -0.02 * h0)
    return sim


@pytest.mark.parametrize("ny,nx,tile,order,sources", [
    (48, 130, (58, 16), 2, True),        # three full chunks of 16 rows by three strips
    (45, 117, (58, 16), 2, False),       # chunks of 15 rows: segments of 4, 4, 4 and 3
    (37, 175, (58, 13), 1, True),        # a last chunk of 11 rows, first order
    (64, 290, (58, 64), 2, True),        # one tall chunk: segments of 16 rows
    (23, 450, (58, 5), 2, True),         # 5-row chunks, the last of 3: a segment without rows
    (9, 464, (58, 9), 1, False),
    (31, 58, (2, 31), 2, True),          # strips of two columns
])
def test_segments_do_not_change_a_bit(ny, nx, tile, order, sources):
    y, x = np.mgrid[0:ny, 0:nx]
    z = 0.003 * x + 0.3 * np.sin(y / 7.0) * np.cos(x / 9.0)
    rain_weight = sources and order == 2
    members = list(range(66))
    groups = {"one": members, "two": members[:27], "alone": members[:1]}
    out = {}
    for name, ms in groups.items():
        sim = _sim(z, ms, order, tile, rain_weight, sources)
        vols = []
        for k in range(5):
            vols.append(sim.step(0.3, 0.3 * k, 2e-5).table.cpu().numpy())
        rate = torch.zeros(len(ms), dtype=torch.float64, pin_memory=True)
        sim.step_rate_async(rate)
        torch.cuda.synchronize()
        out[name] = {f: getattr(sim, f).cpu().numpy().reshape(len(ms), ny, nx) for f in FIELDS}
        out[name]["vols"], out[name]["rate"] = np.stack(vols, axis=1), rate.numpy().copy()
    for name in ("two", "alone"):
        k = len(groups[name])
        for f, a in out[name].items():
            assert np.array_equal(a, out["one"][f][:k]), f"{name}: {f}"
    assert out["one"]["rate"].min() > 0.0 and np.isfinite(out["one"]["h"]).all()
