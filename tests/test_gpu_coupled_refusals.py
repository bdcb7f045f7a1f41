"""What the coupled step's entry point refuses before it queues anything."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grids,nets", [(1, 2), (2, 1), (3, 2)])
def test_sets_of_different_numbers_of_members_are_refused(grids, nets):
    from his_gb300 import _lib, workloads as W
    from his_gb300.boundaries import all_edges
    from his_gb300.config import SolverConfig
    from his_gb300.swe1d import SWE1D
    from his_gb300.swe2d import SWE2D
    cfg, most = SolverConfig(), max(grids, nets)
    storm = W.plain_small()
    two = SWE2D(storm.terrain.z, 0.03, 80.0, cfg, all_edges("closed"), batch=grids)
    one = SWE1D([storm.network] * nets, cfg, inflow=lambda t: np.full(nets, 2.0), stage=lambda t: np.full(nets, 0.5))
    two.set_state(*(torch.full((grids, 81, 100), v, dtype=torch.float64) for v in (0.1, 0.0, 0.0)))
    before = two.h.clone(), one.A.clone(), one.Q.clone()
    # buffers large enough for either set
    ledger = torch.zeros((8, most), dtype=torch.float64, device="cuda")
    rates = torch.full((2 * most,), -7.0, dtype=torch.float64, device="cuda")
    forcing = np.full((most, 1, 2), 0.5)
    params = (_lib.StepParams * most)()
    for m in range(most):
        params[m].dt = 0.1
    s = torch.cuda.current_stream().cuda_stream
    rc = two._lib.his_coupled_step_async(two._handle, one._handle, 0.1, 1, params, _lib.as_p(forcing), ledger.data_ptr(),
                                         rates.data_ptr(), s, torch.cuda.Stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == _lib.HIS_ERR_BAD_ARG and "same number of members" in _lib.last_error()
    assert not ledger.any() and bool((rates == -7.0).all())
    assert torch.equal(two.h, before[0]) and torch.equal(one.A, before[1]) and torch.equal(one.Q, before[2])
