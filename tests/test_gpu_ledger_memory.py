"""A ledger that was device memory once and is not any more is refused, not written to."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_freed_ledger_is_refused():
    from his_gb300 import _lib, workloads as W
    from his_gb300.assembly import build_engine
    eng = build_engine(W.plain_small(), dtype=torch.float64)
    two, one = eng.two, eng.one
    s = torch.cuda.current_stream().cuda_stream
    # an allocation of its own, so that giving it back unmaps it
    torch.cuda.synchronize()
    big = torch.zeros(48 << 20, dtype=torch.float64, device="cuda")
    ledger = big.data_ptr()
    rates = torch.zeros(2, dtype=torch.float64, device="cuda")
    forcing = np.full((1, 1, 2), 0.5)
    params = two.step_params(0.1, 0.0, 0.0)
    calls = {
        "grid": lambda: two._lib.his_grid_step_ledger_async(two._handle, params, ledger, s),
        "network": lambda: two._lib.his_net_step_ledger_async(one._handle, 0.1, 1, _lib.as_p(forcing), ledger, s),
        "coupled": lambda: two._lib.his_coupled_step_async(two._handle, one._handle, 0.1, 1, params, _lib.as_p(forcing),
                                                           ledger, rates.data_ptr(), s, torch.cuda.Stream().cuda_stream),
    }
    for _ in range(3):
        for name, call in calls.items():
            assert call() == 0, name
    torch.cuda.synchronize()
    h = two.h.clone()
    del big
    torch.cuda.empty_cache()
    for name, call in calls.items():
        assert call() == _lib.HIS_ERR_BAD_ARG and "device memory" in _lib.last_error(), name
    torch.cuda.synchronize()
    assert torch.equal(two.h, h)
