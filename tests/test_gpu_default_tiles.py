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
