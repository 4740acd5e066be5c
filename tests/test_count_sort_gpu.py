"""The batch's sort of kept boxes reads their number on the device and works on
as many tiles as they fill.  One workspace over steps that keep many boxes, a
few, none and many again (what an earlier step left behind the live tiles must
not matter), 32- and 64-bit keys; lists equal the per-scene path's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes_n", [4, 260])  # up to 256 scenes the keys have 32 bits
def test_reused_workspace(cuda_device, scenes_n):
    import torch
    from p2cccd_b200 import scenes
    from p2cccd_b200.batch import BatchPipeline

    lon, rings = (120, 96) if scenes_n == 4 else (14, 10)
    v, f = scenes.uv_sphere(lon, rings)
    e = scenes.unique_edges(f)
    batch = []
    for i in range(scenes_n):
        jitter = lambda g=np.random.default_rng(i): g.normal(0.0, 1e-3, v.shape)  # noqa: E731
        batch.append(scenes.combine([(v + jitter(), v + jitter(), f, e), (v + jitter(), v + jitter(), f, e)]))
    a = BatchPipeline(batch, cuda_device, thickness=0.05)
    b = BatchPipeline(batch, cuda_device, thickness=0.05, broad="per_scene")
    caps = [1 << 18 if scenes_n == 4 else 1 << 12] * scenes_n
    a._alloc(caps, caps)
    b._alloc(caps, caps)
    t0, t1 = a.v_t0.clone(), a.v_t1.clone()
    apart = torch.zeros_like(t0)  # moves the second sphere of every scene along the diagonal
    for i, s in enumerate(batch):
        rows = np.repeat((s["v_obj"] == 1).astype(np.float64), 3)
        apart[int(a.v_off[i]):int(a.v_off[i]) + rows.size] = torch.from_numpy(rows).to(cuda_device)
    found, kept = [], []
    for shift in (1.15, 1.42, 3.0, 1.15):  # corners of the envelopes meet, fewer, none, as before
        for p in (a, b):
            p.update_positions(t0 + shift * apart, t1 + shift * apart)
            p.candidates()
        ca, cb = a.read_counts(), b.read_counts()
        assert np.array_equal(ca[:, :3], cb[:, :3])
        assert (ca[:, :2] <= np.array(caps)[:, None]).all()
        for i in range(scenes_n):
            for got, want in zip(a.pairs(i), b.pairs(i)):
                np.testing.assert_array_equal(got, want)
        found.append(int(ca[:, :2].sum()))
        kept.append(int((ca[:, 3] >> 40).sum()))
    assert found[0] == found[3] > 1000 and found[2] == 0
    assert kept[0] == kept[3] > 40000 and 0 < kept[1] < kept[0] / 2 and kept[2] == 0
