"""The float64 2-D step's sub-tiles at the sizes where their indexing can go wrong: one
cell, one past and one short of a sub-tile, last strips narrower and last chunks lower
than the sub-tile the shared memory is sized for, every edge kind, first and second
order, and depths inside the desingularised range."""
import numpy as np
import pytest
import torch

import harness as H

pytestmark = pytest.mark.gpu


def _case(ny, nx, order, flux, h_dry):
    from his_gb300.boundaries import EdgeBC
    from his_gb300.config import SolverConfig
    rng = np.random.default_rng(1000 * ny + nx)
    y, x = np.mgrid[0:ny, 0:nx]
    z = 0.01 * x + 0.4 * np.sin(y / 5.0) * np.cos(x / 7.0) + 0.05 * rng.standard_normal((ny, nx))
    h = np.clip(0.3 - z, 0.0, None) + np.where(rng.random((ny, nx)) < 0.3, 10.0 ** rng.uniform(-6, -2, (ny, nx)), 0.0)
    f = dict(z=z, n=0.02 + 0.03 * rng.random((ny, nx)), S=0.003 * rng.random((ny, nx)),
             horton=(2e-5 + 1e-5 * rng.random((ny, nx)), 2e-6 * np.ones((ny, nx)), 1e-3 * np.ones((ny, nx)), 5.0),
             rw=0.5 + rng.random((ny, nx)), h=h, hu=0.3 * h * rng.standard_normal((ny, nx)),
             hv=0.3 * h * rng.standard_normal((ny, nx)))
    bcs = {"west": EdgeBC("discharge", 0.2), "east": EdgeBC("stage", 0.25), "south": EdgeBC("transmissive"),
           "north": EdgeBC("closed")}
    return f, bcs, SolverConfig(spatial_order=order, flux=flux, h_dry=h_dry)


# strip widths and chunk heights around the 58 x 16 sub-tile: 13-row last chunk of 24-row
# chunks split into 12-row sub-tiles, 55-column last strip of 60-column strips, ...
@pytest.mark.parametrize("ny,nx,tile", [(1, 1, (58, 16)), (1, 3, (2, 1)), (17, 59, (58, 16)), (16, 58, (58, 16)),
                                        (37, 115, (60, 24)), (33, 117, (117, 33)), (5, 120, (1, 3))])
@pytest.mark.parametrize("order,flux,h_dry", [(2, "hllc", 1e-3), (2, "hll", 1e-6), (1, "hllc", 1e-3)])
def test_float64_step_at_sub_tile_edges(ny, nx, tile, order, flux, h_dry):
    from his_gb300.infiltration import Horton
    from his_gb300.swe2d import SWE2D
    from oracle.oracle import OracleSWE2D
    f, bcs, cfg = _case(ny, nx, order, flux, h_dry)

    def sim(tile):
        s = SWE2D(f["z"], f["n"], 9.0, cfg, bcs, storage=f["S"], horton=Horton(*f["horton"]), rain_weight=f["rw"],
                  dy=11.0, tile=tile)
        s.set_state(f["h"], f["hu"], f["hv"])
        return s
    a, b = sim(tile), sim((1, 1))
    o = OracleSWE2D(f["z"], f["n"], 9.0, cfg, bcs, storage=f["S"], horton=f["horton"], rain_weight=f["rw"], dy=11.0)
    o.set_state(f["h"], f["hu"], f["hv"])
    t = 0.0
    for _ in range(3):
        dt = 0.8 * o.max_dt()
        assert a.max_dt() == b.max_dt() == pytest.approx(o.max_dt(), rel=1e-12)
        va, vb = a.step(dt, t, 2e-5), b.step(dt, t, 2e-5)
        o.step(dt, t, 2e-5)
        t += dt
        # the decomposition changes no cell's arithmetic, only the order of the totals
        for name in ("h", "hu", "hv", "s_filled", "infil_cum"):
            assert torch.equal(getattr(a, name), getattr(b, name)), name
            d = H.max_abs(getattr(a, name).cpu().numpy(), getattr(o, name)[0])
            assert d <= 1e-12, f"{name} differs from the oracle by {d}"
        assert torch.allclose(va.table, vb.table, rtol=1e-12, atol=1e-12)


def test_float64_faces_in_their_own_kernel_give_the_fused_kernel_s_bits():
    """A set with room for its faces (40,000 cells and more) computes each face once, in two
    kernels per stage; a smaller set, and the allocation-free step at any size, in one fused
    kernel.  A 205 x 199 grid in 58 x 16 chunks against the allocation-free step's twin of it
    and against a batch of three such members: state and totals bit for bit."""
    import ctypes as C
    from his_gb300 import _lib
    from his_gb300.infiltration import Horton
    from his_gb300.swe2d import SWE2D
    f, bcs, cfg = _case(205, 199, 2, "hllc", 1e-3)
    mk = lambda B: SWE2D(f["z"], f["n"], 9.0, cfg, bcs, storage=f["S"], horton=Horton(*f["horton"]), rain_weight=f["rw"],
                         dy=11.0, batch=B)
    one, many = mk(None), mk(3)
    one.set_state(f["h"], f["hu"], f["hv"])
    many.set_state(f["h"], f["hu"], f["hv"])
    names = ("h", "hu", "hv", "s_filled", "infil_cum")
    twin = {k: getattr(one, k).clone() for k in names}
    d = _lib.GridDesc.from_buffer_copy(one._descs[0])
    d.h, d.hu, d.hv, d.s_filled, d.infil_cum = (twin[k].data_ptr() for k in names)
    ccfg, t = _lib.solver_cfg(cfg), 0.0
    for _ in range(3):
        dt = 0.8 * one.max_dt()
        v = one.step(dt, t, 2e-5)
        many.step(dt, t, 2e-5)
        got = np.zeros(5)
        _lib.check(one._lib.his_grid_step_noalloc(one.prec, C.byref(ccfg), C.byref(d), one.step_params(dt, t, 2e-5),
                                                  _lib.as_p(got), _lib.stream_handle()), "his_grid_step_noalloc")
        t += dt
        assert np.array_equal(got, v.table[0].cpu().numpy())
        for k in names:
            assert torch.equal(getattr(one, k), twin[k]), k
            assert all(torch.equal(getattr(many, k)[b], twin[k]) for b in range(3)), k


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ny,nx", [(1, 40), (40, 1), (23, 61)])
def test_float64_contact_side_on_closed_thin_films(ny, nx, order):
    # depths around 1e-9, where the contact speed's sign is taken from its quotient and above
    # which from the mass flux, all above the dry threshold and in closed walls (an inflow of
    # given discharge into a film would move at 1e8 m/s).  Values stay under 1e-5 at speeds
    # under 1: about a hundred roundings of them, 100 x 1e-5 x 1.1e-16, are well within 1e-15
    from his_gb300.boundaries import EdgeBC
    from his_gb300.config import SolverConfig
    from his_gb300.swe2d import SWE2D
    from oracle.oracle import OracleSWE2D
    rng = np.random.default_rng(7 * ny + nx)
    z, h = 1e-9 * rng.standard_normal((ny, nx)), 10.0 ** rng.uniform(-12, -6, (ny, nx))
    cfg = SolverConfig(spatial_order=order, flux="hllc", h_dry=1e-13, kp_eps=1e-60)
    bcs = {e: EdgeBC("closed") for e in ("west", "east", "south", "north")}
    s, o = (C(z, 0.03 * np.ones((ny, nx)), 9.0, cfg, bcs, dy=11.0) for C in (SWE2D, OracleSWE2D))
    for x in (s, o):
        x.set_state(h, 0.5 * h, -0.25 * h)
    for k in range(3):
        s.step(0.1, 0.1 * k, 0.0)
        o.step(0.1, 0.1 * k, 0.0)
        for name in ("h", "hu", "hv"):
            d = H.max_abs(getattr(s, name).cpu().numpy(), getattr(o, name)[0])
            assert d <= 1e-15, f"{name} differs from the oracle by {d}"


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nx", [511, 512, 513])
def test_totals_around_the_split_of_finalize(nx, dtype):
    # members of 512 chunks and more are totalled by eight CTAs.  The totals of 1 x nx cells in
    # one-cell and in 58-cell chunks differ by the order of at most 513 float64 adds, and in
    # float32 by that of a chunk's 58 partial sums
    from his_gb300.swe2d import SWE2D
    f, bcs, cfg = _case(1, nx, 2, "hllc", 1e-3)
    sims = [SWE2D(f["z"], f["n"], 9.0, cfg, bcs, storage=f["S"], rain_weight=f["rw"], dy=11.0, tile=t, dtype=dtype)
            for t in ((1, 1), (58, 16))]
    for s in sims:
        s.set_state(f["h"], f["hu"], f["hv"])
    assert sims[0].max_dt() == sims[1].max_dt()
    dt = 0.5 * sims[1].max_dt()
    a, b = (s.step(dt, 0.0, 2e-5) for s in sims)
    assert torch.equal(sims[0].h, sims[1].h)
    rel = 1e-12 if dtype == torch.float64 else 58 * 2.0 ** -24
    assert torch.allclose(a.table, b.table, rtol=rel, atol=1e-12)
