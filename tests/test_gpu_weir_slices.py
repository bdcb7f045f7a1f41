"""The weir exchange where its slicing can go wrong: no shared 2-D cell and many, fewer links
than CTAs, more than a thread fetches ahead, all links on one channel cell.  Against the
method in numpy (coupling.py:73-124)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(cfg, tp, sec, A, h, hu, hv, z2, area, c1, c2, length, dt):
    b, m, yb, ts = (sec[k] for k in ("b", "m", "yb", "ts"))
    ab = yb * (b + m * yb)
    y = np.where(A <= ab, 2 * A / (b + np.sqrt(b * b + 4 * m * A)), yb + (A - ab) / ts)
    plan = (np.where(y <= yb, b + 2 * m * y, ts) * tp.dx)[c1]
    e1, e2 = (tp.z + y)[c1], z2[c2] + h[c2]
    up, dn = np.maximum(e1, e2), np.minimum(e1, e2)
    du, dd = np.maximum(up - tp.zbank[c1], 0), np.maximum(dn - tp.zbank[c1], 0)
    r = np.where(du > 0, dd / np.where(du > 0, du, 1), 0)
    q = cfg.weir_cw * length * du ** 1.5 * np.maximum(1 - r ** 1.5, 0) ** 0.385
    V = np.minimum(q * dt, cfg.exchange_relax * (up - dn) / (1 / area + 1 / plan))
    into = e2 > e1
    take2, take1 = np.zeros_like(h), np.zeros_like(A)
    np.add.at(take2, c2, np.where(into, V, 0))
    np.add.at(take1, c1, np.where(into, 0, V))
    have2 = cfg.exchange_limit * h * area
    have1 = cfg.exchange_limit * np.maximum(A - ab, 0) * tp.dx
    f = lambda t, a: np.where(t > a, a / np.where(t > 0, t, 1), 1.0)
    V = np.where(into, V * f(take2, have2)[c2], -V * f(take1, have1)[c1])
    d2, d1 = np.zeros_like(h), np.zeros_like(A)
    np.add.at(d2, c2, V)
    np.add.at(d1, c1, V)
    hn = h - d2 / area
    keep = np.where(h > 0, np.minimum(hn / np.where(h > 0, h, 1), 1), 0)
    on = np.zeros(h.shape, bool)
    on[c2] = True
    return V, np.where(on, hn, h), np.where(on, hu * keep, hu), np.where(on, hv * keep, hv), A + d1 / tp.dx


# Absolute tolerance of one link's volume [m^3].  float64: volumes of up to 1e3 m^3 from levels
# of tens of metres (ulp 7e-15) times plan areas of 800 m^2.  float32: levels of up to 64 m
# (ulp 3.8e-6, up to 8e-6 in a difference of two) times half the 2-D cell's 1600 m^2, doubled
# for the donor limits' factors.  States take their links' errors over their areas.
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 2e-11), (torch.float32, 2e-2)])
@pytest.mark.parametrize("n_links,n_cells2d,one_cell", [(1, 40, False), (5, 3, False), (700, 5000, False),
                                                        (1700, 300, False), (1600, 5000, True)])
def test_exchange_matches_the_method_for_any_sharing_of_cells(dtype, tol, n_links, n_cells2d, one_cell):
    from his_gb300 import workloads as W
    from his_gb300.boundaries import all_edges
    from his_gb300.config import SolverConfig
    from his_gb300.coupling import exchange, links_from_cells
    from his_gb300.swe1d import SWE1D
    from his_gb300.swe2d import SWE2D
    from his_gb300.topology import build_topology, sections
    rng = np.random.default_rng(n_links + n_cells2d)
    ter = W.make_terrain(200, 163, 40.0, 18, "weir-slices", "triple")
    net, cfg = W.make_network(ter, "triple"), SolverConfig()
    tp = build_topology(net)
    sec = sections(tp, cfg.slot_width_frac)
    one = SWE1D(net, cfg)
    y = sec["yb"] * rng.uniform(0.6, 1.2, tp.n_cells)
    yt = np.minimum(y, sec["yb"])
    A = yt * (sec["b"] + sec["m"] * yt) + sec["ts"] * np.maximum(y - sec["yb"], 0.0)
    interior = np.nonzero(tp.kind <= 1)[0]
    c1 = np.full(n_links, interior[3]) if one_cell else rng.choice(interior, n_links)
    pool = rng.permutation(ter.nx * ter.ny)[:n_cells2d]
    c2 = pool[:n_links] if n_links <= n_cells2d else rng.choice(pool, n_links)
    # beds near the banks they are linked to, so that links overtop in both directions
    z = ter.z.reshape(-1).copy()
    z[c2] = tp.zbank[c1] + rng.uniform(-0.3, 0.1, n_links)
    two = SWE2D(z.reshape(ter.z.shape), 0.03, ter.dx, cfg, all_edges("closed"), dtype=dtype)
    h = np.where(rng.random(z.size) < 0.2, 0.0, rng.uniform(0.0, 0.8, z.size))
    st = [torch.as_tensor(a).to(dtype) for a in (h, h * rng.normal(size=z.size), h * rng.normal(size=z.size))]
    two.set_state(*(a.reshape(ter.z.shape) for a in st))
    one.A = A
    length = rng.uniform(20.0, 60.0, n_links)
    links = links_from_cells(one, two, c1, c2, length)
    V = exchange(one, two, links, 0.7, cfg).cpu().numpy()
    z2 = two.z.double().cpu().numpy().reshape(-1)
    want = _expected(cfg, tp, sec, A, *(a.double().numpy() for a in st), z2, ter.dx ** 2, c1, c2, length, 0.7)
    got = (V,) + tuple(getattr(two, k).double().cpu().numpy().reshape(-1) for k in ("h", "hu", "hv")) + \
        (one.A.cpu().numpy(),)
    assert np.abs(want[0]).max() > 0
    shared, per_cell = np.bincount(c2).max(), np.bincount(c1).max()
    err_h = shared * tol / ter.dx ** 2 + (1e-6 if dtype == torch.float32 else 1e-15)
    fast = float((st[1].abs() / st[0].clamp(min=1e-30) * (st[0] > 0)).max().clamp(min=1.0)) + \
        float((st[2].abs() / st[0].clamp(min=1e-30) * (st[0] > 0)).max())
    bound = {"V": tol, "h": err_h, "hu": fast * err_h, "hv": fast * err_h, "A": per_cell * tol / tp.dx.min()}
    for name, a, w in zip(("V", "h", "hu", "hv", "A"), got, want):
        d = float(np.abs(a - w).max())
        assert d <= bound[name], (name, d, bound[name])
    total = links.exchanged()[0]
    assert abs(total[0] - np.maximum(want[0], 0).sum()) <= n_links * tol
    assert abs(total[1] - np.maximum(-want[0], 0).sum()) <= n_links * tol
