"""Engine steps in one graph against the same steps one graph each.

Within a graph the accounting of a step and the pre-step of the next are one kernel; a
graph of one step launches them apart.  Both must leave the same bits: states,
accumulators, clocks, peaks, output series and their ledgers, with members that end
before the others.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,interval,couple", [
    ("fp64", 1, 120.0, True), ("fp64", 3, None, True), ("fp64", 2, 120.0, False),
    ("fp32", 1, 120.0, True), ("fp32", 5, 90.0, True), ("fp32", 32, None, True), ("fp32", 33, None, True),
    ("fp32", 2, None, False),
])
def test_steps_in_one_graph_equal_single_steps(precision, n, interval, couple):
    from his_gb300 import workloads as W
    from his_gb300.config import SolverConfig
    from his_gb300.engine import FloodEngine
    engines = []
    for graph_steps in (1, 8):
        storms = [W.plain_small() for _ in range(n)]
        for k, s in enumerate(storms):
            s.t_end = 330.0 + 40.0 * k                   # members end one after the other
        engines.append(FloodEngine(storms, SolverConfig(slot_width_frac=storms[0].slot_width_frac),
                                   precision=precision, tile=(58, 16), graph_steps=graph_steps, couple=couple,
                                   track_peaks=True, output_interval=interval))
    for steps in (24, 200):                              # still running; most members ended
        for fe in engines:
            fe.advance(steps)
        torch.cuda.synchronize()
        a, b = engines
        for name in ("h", "hu", "hv") + (("A", "Q") if couple else ()):
            for x, y in zip(getattr(a, name), getattr(b, name)):
                assert torch.equal(x, y), f"{name} after {steps}"
        for m, (x, y) in enumerate(zip(a.reports(), b.reports())):
            assert (x.steps, x.t, x.status) == (y.steps, y.t, y.status), f"member {m}"
            assert np.array_equal(np.asarray(x.acc), np.asarray(y.acc)), f"member {m}: accumulators"
            for f in ("dt_min", "dt_max", "n_sub_max", "n_clamped", "outputs"):
                if hasattr(x, f):
                    assert getattr(x, f) == getattr(y, f), f"member {m}: {f}"
    assert engines[1].reports()[0].status == 1
    if not interval:
        return
    for x, y in zip(engines[0].flood_results(), engines[1].flood_results()):
        for key in ("depth_series", "u", "v", "times", "depth_max"):
            p, q = getattr(x, key, None), getattr(y, key, None)
            if torch.is_tensor(p):
                assert torch.equal(p, q), key
        assert x.extras["ledger"] == y.extras["ledger"]
