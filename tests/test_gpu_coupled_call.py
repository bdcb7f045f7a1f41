"""The coupled step's one native call against the calls it joins.

CoupledEngine.step issues the 2-D step, the 1-D substeps beside it and the next step's
1-D rates through his_coupled_step_async (coupling.py:212-227).  The same entry points
called one after the other on one stream must leave the same bits.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n_sub", [1, 3])
def test_one_call_equals_the_separate_calls(dtype, n_sub):
    from his_gb300 import workloads as W
    from his_gb300.assembly import build_engine
    from his_gb300.coupling import exchange
    storm = W.plain_small()
    a, b = build_engine(storm, dtype=dtype), build_engine(storm, dtype=dtype)
    dt = 0.5 * a.two.max_dt()
    ledger = b.mb.device_ledger(b.two.device)
    t = 0.0
    for _ in range(6):
        a.step(t, storm.t_end, dt=dt, n_sub=n_sub)
        exchange(b.one, b.two, b.links, dt, b.cfg, volumes=False)
        b.two.step_ledger(dt, t, b.rain(t), None, ledger.data_ptr())
        b.one.substeps_ledger(dt, t, n_sub, ledger.data_ptr())
        t += dt
    torch.cuda.synchronize()
    for f in ("h", "hu", "hv"):
        assert torch.equal(getattr(a.two, f), getattr(b.two, f)), f
    for f in ("A", "Q"):
        assert torch.equal(getattr(a.one, f), getattr(b.one, f)), f
    assert torch.equal(a.mb.device_ledger(a.two.device), ledger)
    # the rates reduced ahead are those of the state the step left
    got = a._rates[a.two.B:].numpy().copy()
    rate, wet = b.one.member_rates()
    assert np.array_equal(got.reshape(-1, 2)[:, 0], rate) and np.array_equal(got.reshape(-1, 2)[:, 1] > 0, wet > 0)


def test_too_few_edge_values_are_refused():
    # records are laid out once and refilled: a short list must not leave old edge values in
    from his_gb300 import workloads as W
    from his_gb300.assembly import build_engine
    two = build_engine(W.plain_small(), dtype=torch.float32).two
    before = two.h.clone()
    for edges in ([], [0.0, 0.0, 0.0]):
        with pytest.raises(ValueError):
            two.step(0.1, 0.0, 0.0, edges)
    torch.cuda.synchronize()
    assert torch.equal(two.h, before)
