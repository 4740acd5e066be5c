"""Calls on a stream that owns part of the SMs (a green context of 16): no
launch needs all SMs of the device at once.  Pair lists with rows of several
tiles, a batch of them and candidate groups of several tiles, against the same
calls on the whole device.  In a child process, so that the partition ends
with it."""
from __future__ import annotations

import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

CHILD = r"""
import json, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/p2c-ccd_b200", sys.argv[1] + "/tests"]
import numpy as np
import torch
from dense_inputs import make_rows
from test_batch_windows_gpu import _sheet_over_quad
from p2cccd_b200.batch import BatchPipeline
from p2cccd_b200.dense_groups import DenseGroupEarlyStop, _query_bits, upload
from p2cccd_b200.scene import ScenePipeline

dev = torch.device("cuda:0")
scene = ScenePipeline(_sheet_over_quad(120), dev, vf_capacity=1 << 17, ee_capacity=1 << 17)
scene.step_checked()
batch = BatchPipeline([_sheet_over_quad(n) for n in (120, 20, 90)], dev)
batch.step_checked()
rows = make_rows(50000, 3)
rows["query_id"] = np.random.default_rng(3).permutation(np.repeat([1, 2, 3], [33000, 16000, 1000])).astype(np.uint64)
up, bits = upload(rows, dev), _query_bits(rows["query_id"])
groups = DenseGroupEarlyStop(50000, dev)

def calls():
    for t in (scene.vf_pairs, scene.ee_pairs, batch.vf_pairs, batch.ee_pairs):
        t.zero_()
    scene.step()
    batch.step()
    groups.run(up, 50000, query_bits=bits)

def outputs():
    torch.cuda.synchronize()
    return [np.concatenate([a.view(np.uint8).ravel() for a in (*scene.pairs(), *scene.results())]),
            np.concatenate([a.view(np.uint8).ravel() for i in range(3) for a in (*batch.pairs(i), *batch.results(i))]),
            groups.stats.cpu().numpy()]

calls()
want = outputs()
try:
    from cuda.bindings import driver as d
except ImportError:
    print(json.dumps({"skip": "no driver bindings"}))
    sys.exit(0)

def ok(r):
    if int(r[0]) != 0:
        print(json.dumps({"skip": "SM partitions are not available: %s" % r[0]}))
        sys.exit(0)
    return r[1] if len(r) == 2 else r[1:]

res = ok(d.cuDeviceGetDevResource(0, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
part, n, _ = ok(d.cuDevSmResourceSplitByCount(1, res, 0, 16))
desc = ok(d.cuDevResourceGenerateDesc(part[:1], 1))
green = ok(d.cuGreenCtxCreate(desc, 0, int(d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM)))
stream = ok(d.cuGreenCtxStreamCreate(green, int(d.CUstream_flags.CU_STREAM_NON_BLOCKING), 0))
with torch.cuda.stream(torch.cuda.ExternalStream(int(stream))):
    calls()
got = outputs()
print(json.dumps({"sms": int(part[0].sm.smCount), "same": [bool(np.array_equal(a, b)) for a, b in zip(got, want)]}))
"""


def test_calls_on_a_partition_of_the_sms(cuda_device):
    r = subprocess.run([sys.executable, "-c", CHILD, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    if "skip" in out:
        pytest.skip(out["skip"])
    assert out["sms"] < 64 and out["same"] == [True, True, True], out
