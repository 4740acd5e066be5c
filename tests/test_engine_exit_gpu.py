"""The end of a launch: idle warps hold a ticket each and wait for a node or
for the last query.  A warp's lanes leave that wait together, on one lane's
read of the finished count, as everything after it works on whole warps.  No
run can show a lane that left alone, so this covers the path: many launches
whose last queries are deep trees shared among warps, byte for byte against
the CPU oracle (no tolerance)."""
from __future__ import annotations

import numpy as np
import pytest

from test_engine_edges_gpu import _bytes, _grazing

pytestmark = pytest.mark.gpu


def test_waiting_warps_leave_together(cuda_device, oracle_mod):
    import torch
    from p2cccd_b200 import certify

    cfg = (1e-12, 1e-6, 13)
    rec = _grazing(40, 0.3, 1e-9)
    cpu, st, _ = oracle_mod.eval_batch(rec, 0.0, 1.0, *cfg)
    assert st.sum() == 0
    ws = certify.Workspace(torch.device(cuda_device))
    shared = 0
    for k in range(200):
        n = 1 + k % 40
        out = certify.certify_batch(certify.records_to_device(rec[:n]), 1, 0.0, 1.0, certify.CertConfig(*cfg),
                                    workspace=ws)
        torch.cuda.synchronize()
        stats = ws.stats()
        assert stats["error_word"] == 0 and stats["queries"] == n
        shared += stats["donations"]
        np.testing.assert_array_equal(_bytes(certify.results_to_numpy(out)), _bytes(cpu[:n]))
    assert shared > 0


def test_pool_ring_laps(cuda_device, oracle_mod):
    """Deep trees that publish more nodes than the ring of 16,384 places holds
    (45,000 measured), so that places are used again."""
    import torch
    from p2cccd_b200 import certify

    cfg = (1e-12, 1e-6, 16)
    rec = _grazing(30, 0.3, 1e-9)
    cpu, st, _ = oracle_mod.eval_batch(rec, 0.0, 1.0, *cfg)
    assert st.sum() == 0
    ws = certify.Workspace(torch.device(cuda_device))
    out = certify.certify_batch(certify.records_to_device(rec), 1, 0.0, 1.0, certify.CertConfig(*cfg), workspace=ws)
    torch.cuda.synchronize()
    stats = ws.stats()
    assert stats["error_word"] == 0 and stats["donations"] > 16384
    np.testing.assert_array_equal(_bytes(certify.results_to_numpy(out)), _bytes(cpu))
