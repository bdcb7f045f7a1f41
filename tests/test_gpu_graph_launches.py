"""Steps launched as graphs against the same kernels launched one by one (his_grid_step), and
the coupled graph when what it was captured for changes."""
import numpy as np
import pytest
import torch

import test_gpu_ledger_graph as L

pytestmark = pytest.mark.gpu


def test_graphs_of_member_parts_equal_plain_launches():
    from his_gb300 import _lib
    from his_gb300.massbalance import MassBalance
    sims = {k: L._batch() for k in ("plain", "ledger", "async")}
    tiles = L.B * -(-L.NX // L.TILE[0]) * -(-L.NY // L.TILE[1])
    assert int(sims["plain"]._lib.his_engine_default_chains(L.B, tiles)) >= 2      # the step forks member parts
    ledger = MassBalance(sims["plain"].device, np.zeros(L.B)).device_ledger(sims["plain"].device)
    sums, vols = np.zeros((L.B, 5)), np.zeros((L.B, 5))
    rain, dt = 2e-5 * (1.0 + np.arange(L.B) / L.B), 0.4
    for k in range(6):
        t = k * dt
        p = sims["plain"]
        _lib.check(p._lib.his_grid_step(p._handle, p.step_params(dt, t, rain), _lib.as_p(vols), _lib.stream_handle()),
                   "his_grid_step")
        sims["ledger"].step_ledger(dt, t, rain, None, ledger.data_ptr())
        v = sims["async"].step(dt, t, rain).table.cpu().numpy()
        assert np.array_equal(v, vols), k
        sums += vols
        for name in ("ledger", "async"):
            for f in L.FIELDS:
                assert torch.equal(getattr(sims[name], f), getattr(p, f)), (name, f, k)
    s, led = sums.T, ledger.cpu().numpy()
    for row, term in ((L.LG_RAIN, 2), (L.LG_INFIL, 3), (L.LG_BND2_IN, 0), (L.LG_BND2_OUT, 1), (L.LG_CLIP2, 4)):
        assert np.array_equal(led[row], s[term]), row


def _coupled(n):
    from his_gb300 import workloads as W
    from his_gb300.assembly import build_engine, build_engine_batch
    if n == 1:
        return build_engine(W.plain_small(), dtype=torch.float64)
    first = W.plain_small()
    return build_engine_batch([first] + [W.Storm(**{**vars(first), "key": f"m{k}", "manning": 0.03 + 0.0005 * k})
                                         for k in range(1, n)], dtype=torch.float32, tile=(58, 16))


def _separately(eng, dt, t, ledger, n_sub):
    eng.two.step_ledger(dt, t, eng.rain(t), None, ledger.data_ptr())
    eng.one.substeps_ledger(dt, t, n_sub, ledger.data_ptr())


def _in_one(eng, net, dt, t, ledger, rates, n_sub, side):
    from his_gb300 import _lib
    from his_gb300.boundaries import edge_values
    params = eng.two.step_params(dt, t, eng.rain(t), edge_values(eng.two.bcs, t))
    f = net.substep_forcing(dt, t, n_sub)
    _lib.check(eng.two._lib.his_coupled_step_async(eng.two._handle, net._handle, dt, n_sub, params, _lib.as_p(f),
                                                   ledger.data_ptr(), rates.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream, side.cuda_stream), "coupled")


def _same(a, b, one, la, lb, rates):
    torch.cuda.synchronize()
    for f in ("h", "hu", "hv"):
        assert torch.equal(getattr(a.two, f), getattr(b.two, f)), f
    for f in ("A", "Q"):
        assert torch.equal(getattr(one, f), getattr(b.one, f)), f
    assert torch.equal(la, lb)
    rate, wet = b.one.member_rates()
    got = rates.cpu().numpy().reshape(-1, 2)
    assert np.array_equal(got[:, 0], np.atleast_1d(rate)) and np.array_equal(got[:, 1] > 0, np.atleast_1d(wet) > 0)


@pytest.mark.parametrize("n", [1, 48])              # 48: two member parts beside the 1-D side
def test_the_coupled_graph_follows_its_arguments(n):
    from his_gb300.swe1d import SWE1D
    a, b = _coupled(n), _coupled(n)
    if n > 1:
        assert int(a.two._lib.his_engine_default_chains(n, n * 2 * 6)) >= 2
    dt, side = 0.25 * a.two.max_dt(), torch.cuda.Stream()
    zeros = lambda: torch.zeros((8, n), dtype=torch.float64, device="cuda")
    rates = lambda: torch.full((2 * n,), -3.0, dtype=torch.float64, device="cuda")
    others = _coupled(n)                             # (its network is the second one)
    ledger, rate, t = zeros(), rates(), 0.0
    first, one = (ledger, rate), a.one
    for change in ("none", "ledger", "rates", "network", "ledger and rates back"):
        if change == "ledger":
            ledger = zeros()
        elif change == "rates":
            rate = rates()
        elif change == "network":
            others.one.A, others.one.Q = one.A.clone(), one.Q.clone()
            one = others.one
        elif change != "none":
            ledger, rate = first
        want = ledger.clone()
        for _ in range(4):
            _in_one(a, one, dt, t, ledger, rate, 2, side)
            _separately(b, dt, t, want, 2)
            t += dt
        _same(a, b, one, ledger, want, rate)
