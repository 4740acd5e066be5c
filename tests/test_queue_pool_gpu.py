"""The work-queue certifier shares deep trees among warps, with a caller's
workspace and with the library's own scratch: certificates byte for byte
against the CPU oracle (no tolerance), and nodes handed to other warps."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_engine_edges_gpu import _bytes, _grazing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("items,per,depth", [(1, 1, 15), (200, 6, 11), (13000, 1, 6)])
def test_deep_work_items(cuda_device, oracle_mod, items, per, depth, static):
    import torch
    from p2cccd_b200 import _lib, records, workloads

    lib = _lib.load()
    n = items * per
    vf = _grazing(n, 0.3, 1e-9)
    ee = workloads.plain_queries(workloads.PlainSpec(n_vf=1, n_ee=n, seed=4))["ee"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).to(cuda_device)  # noqa: E731
    off = dev(np.arange(items + 1, dtype=np.int64) * per)
    of = dev(np.repeat(np.arange(items, dtype=np.int64), per))
    pt, e, t0, t1 = dev(vf), dev(ee), dev(np.zeros(items)), dev(np.ones(items))
    mask = dev(np.full(items, 3, np.uint32))
    out = [torch.zeros((n, 72), dtype=torch.uint8, device=cuda_device) for _ in range(2)]
    certs = torch.zeros((items, records.QUERY_CERTIFICATE_DTYPE.itemsize), dtype=torch.uint8, device=cuda_device)
    stats = torch.zeros(8, dtype=torch.int64, device=cuda_device)
    cfg = (1e-12, 1e-6, depth)
    c = _lib.make_config(*cfg)
    args = [pt.data_ptr(), n, of.data_ptr(), e.data_ptr(), n, of.data_ptr(), items, off.data_ptr(), off.data_ptr(),
            t0.data_ptr(), t1.data_ptr(), mask.data_ptr(), ctypes.byref(c), out[0].data_ptr(), out[1].data_ptr(),
            certs.data_ptr()]
    size = int(lib.p2c_certify_queries_workspace_bytes(items))
    ws = torch.empty(size, dtype=torch.uint8, device=cuda_device)
    stream = torch.cuda.current_stream(cuda_device).cuda_stream
    for _ in range(2):  # the second call on used scratch
        _lib.check(lib.p2c_certify_queries_static(*args, stats.data_ptr(), stream) if static else
                   lib.p2c_certify_queries(*args, ws.data_ptr(), size, stats.data_ptr(), stream))
        torch.cuda.synchronize(cuda_device)
        donations, queries, error = (int(x) for x in stats[3:6])
        assert error == 0 and queries == 2 * n and donations > 0
        for rec, got in ((vf, out[0]), (ee, out[1])):
            cpu, st, _ = oracle_mod.eval_batch(rec, 0.0, 1.0, *cfg)
            assert st.sum() == 0
            np.testing.assert_array_equal(got.cpu().numpy(), _bytes(cpu))
