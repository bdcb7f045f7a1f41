"""The weir exchange inside the resident engine, whose members' pre-steps have one, four or
eight CTAs by precision and by the size of the set.

With links that share 2-D cells across the CTAs' slices and more links per slice than
threads: a member's states and exchanged totals must not depend on the set's size, and a
float64 member's are those of the drop-in coupled step (coupling.py:73-124, 205-230).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N_LINKS, N_CELLS2D, STEPS = 4200, 2500, 3


def _storm():
    """A small storm whose channel stands at its banks beside wet 2-D cells: the storm, its
    links and the states (depth, wetted area)."""
    from his_gb300 import workloads as W
    from his_gb300.topology import build_topology, sections
    rng = np.random.default_rng(5)
    storm = W.plain_small()
    tp = build_topology(storm.network)
    sec = sections(tp, storm.slot_width_frac)
    c1 = rng.choice(np.nonzero(tp.kind <= 1)[0], N_LINKS)
    c2 = rng.choice(rng.permutation(storm.terrain.z.size)[:N_CELLS2D], N_LINKS)
    z = storm.terrain.z.reshape(-1).copy()
    z[c2] = tp.zbank[c1] + rng.uniform(-0.3, 0.1, N_LINKS)
    storm.terrain.z[...] = z.reshape(storm.terrain.z.shape)
    h = np.where(rng.random(z.size) < 0.2, 0.0, rng.uniform(0.0, 0.3, z.size)).reshape(storm.terrain.z.shape)
    A = sec["yb"] * (sec["b"] + sec["m"] * sec["yb"]) * rng.uniform(0.95, 1.05, tp.n_cells)
    return storm, tp, c1, c2, rng.uniform(1.0, 4.0, N_LINKS), h, A


def _engine(n, precision, data):
    from his_gb300 import _lib
    from his_gb300.config import SolverConfig
    from his_gb300.engine import FloodEngine, Member
    storm, tp, c1, c2, length, h, A = data
    uniq, inv = np.unique(c2, return_inverse=True)
    members, zcache = [], {}
    for _ in range(n):
        m = Member(storm, torch.float64 if precision == "fp64" else torch.float32,
                   torch.device("cuda", torch.cuda.current_device()), True, False, zcache)
        m.h.copy_(torch.as_tensor(h))
        m.A.copy_(torch.as_tensor(A))
        m._link_arrays = {
            "cell1d": _lib.host_array(c1, np.int32), "inv": _lib.host_array(inv, np.int32),
            "uniq": _lib.host_array(uniq, np.int64), "zbank": _lib.host_array(tp.zbank[c1], np.float64),
            "length": _lib.host_array(length, np.float64),
            "z2": _lib.host_array(m.z.double().cpu().numpy().reshape(-1)[c2], np.float64)}
        m.n_links = N_LINKS
        members.append(m)
    fe = FloodEngine(members, SolverConfig(slot_width_frac=storm.slot_width_frac), precision=precision, tile=(58, 16))
    fe.advance(STEPS)
    torch.cuda.synchronize()
    moved = np.zeros((n, 2))
    _lib.check(fe._lib.his_links_exchanged(fe._links, _lib.as_p(moved), 0, _lib.stream_handle()), "exchanged")
    return fe, moved


def _state(m):
    return {k: getattr(m, k).cpu() for k in ("h", "hu", "hv", "A", "Q")}


@pytest.mark.parametrize("precision,sizes", [("fp32", (1, 32, 33)), ("fp64", (1, 5))])
def test_a_member_does_not_depend_on_the_size_of_its_set(precision, sizes):
    data = _storm()
    alone, moved = _engine(sizes[0], precision, data)
    want = _state(alone.members[0])
    assert moved.min() > 0.0 and alone.reports()[0].steps == STEPS and torch.isfinite(want["h"]).all()
    for n in sizes[1:]:
        fe, got = _engine(n, precision, data)
        for m in (0, n - 1):
            for k, v in _state(fe.members[m]).items():
                assert torch.equal(v, want[k]), f"{k} of member {m} of {n}"
            assert np.array_equal(got[m], moved[0]), f"totals of member {m} of {n}"


def test_a_float64_member_steps_as_the_drop_in_engine():
    from his_gb300.assembly import build_engine
    from his_gb300.coupling import links_from_cells
    data = _storm()
    storm, tp, c1, c2, length, h, A = data
    eng = build_engine(storm, dtype=torch.float64)
    eng.links = links_from_cells(eng.one, eng.two, c1, c2, length)
    eng.two.set_state(torch.as_tensor(h), torch.zeros(h.shape), torch.zeros(h.shape))
    eng.one.A, eng.one.Q = A, np.zeros_like(A)
    t = 0.0
    for _ in range(STEPS):
        t = eng.step(t, storm.t_end)
    fe, moved = _engine(1, "fp64", data)
    want, r = _state(fe.members[0]), fe.reports()[0]
    assert r.t == t and r.n_sub_max == eng.log.n_sub_max
    for k in ("h", "hu", "hv"):
        assert torch.equal(getattr(eng.two, k).cpu(), want[k]), k
    for k in ("A", "Q"):
        assert torch.equal(getattr(eng.one, k).cpu(), want[k]), k
    assert np.array_equal(eng.links.exchanged()[0], moved[0])
