"""Pair lists put into rows: rows around every size where their order is made
differently (counting, a warp, a block's tile, one merge, several), and lists
that overflow their buffers.  Pair sets are exact."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(k):
    """One triangle whose every vertex sweeps over k small separate ones: each
    of its vertices meets k faces, each of its edges 3 k edges."""
    from p2cccd_b200 import scenes

    g = np.random.default_rng(k)
    at = np.repeat(g.uniform(-1.0, 1.0, (k, 1, 3)), 3, axis=1).reshape(-1, 3)
    small = at + g.normal(0.0, 1e-3, at.shape)
    big = g.normal(0.0, 0.1, (3, 3))
    objs = [(big - 10.0, big + 10.0, np.array([[0, 1, 2]], np.int32)),
            (small, small + g.normal(0.0, 1e-3, small.shape), np.arange(3 * k, dtype=np.int32).reshape(-1, 3))]
    return scenes.combine([(a, b, f, scenes.unique_edges(f)) for a, b, f in objs])


def _expected(k):
    key = lambda a, b: (np.asarray(a, np.uint64) << np.uint64(32)) | np.asarray(b, np.uint64)  # noqa: E731
    vf = np.concatenate([key(v, np.arange(1, k + 1)) for v in range(3)] + [key(np.arange(3, 3 * k + 3), 0)])
    return vf, np.concatenate([key(e, np.arange(3, 3 * k + 3)) for e in range(3)])


@pytest.mark.parametrize("k", [1, 5, 6, 16, 17, 32, 33, 64, 65, 85, 86, 128, 129, 256, 257, 341, 342, 512, 513, 1024, 1025, 2730, 2731, 8192, 8193, 20000])
def test_rows_of_every_length(cuda_device, k):
    from p2cccd_b200.scene import ScenePipeline

    want = _expected(k)
    cap = max(17000, 10 * k)  # past the rank sort
    p = ScenePipeline(_scene(k), cuda_device, vf_capacity=cap, ee_capacity=cap)
    for _ in range(2):
        p.candidates()
        assert p.read_counts() == (len(want[0]), len(want[1]), 0)
        for pairs, w in zip((p.vf_pairs, p.ee_pairs), want):
            got = pairs.cpu().numpy().view(np.uint64)
            np.testing.assert_array_equal(got[:len(w)], w)
            assert (got[len(w):] == np.uint64(2**64 - 1)).all()


@pytest.mark.parametrize("vf_cap,ee_cap", [(17000, 30000), (1, 50000), (60000, 20000)])
def test_rows_of_overflowing_lists(cuda_device, vf_cap, ee_cap):
    from p2cccd_b200.scene import ScenePipeline

    want = _expected(8193)
    p = ScenePipeline(_scene(8193), cuda_device, vf_capacity=vf_cap, ee_capacity=ee_cap)
    p.candidates()
    assert p.read_counts()[:2] == (len(want[0]), len(want[1]))
    for pairs, w in zip((p.vf_pairs, p.ee_pairs), want):
        got = pairs.cpu().numpy().view(np.uint64)
        live = got[:len(w)]
        assert (live[1:] > live[:-1]).all() and np.isin(live, w).all()
        assert (got[len(w):] == np.uint64(2**64 - 1)).all()
