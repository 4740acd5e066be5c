"""The binned broad phase where its grid changes shape, against the oracle's
brute force (pair sets are exact, no tolerance): a few oversized boxes (the
second size class), coordinates far from the origin (the widened columns span
many), flat and fully coincident scenes (one column, one bin), one, three and
more objects than culling handles, single primitives, and pair lists on both
sides of the rank sort's limit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheet(n, cell, z=0.0, seed=0, motion=0.0):
    g = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(n) * cell, np.arange(n) * cell)
    v0 = np.stack([x.ravel(), y.ravel(), np.full(n * n, z)], 1)
    v0 = v0 + g.normal(0, 0.05 * cell, v0.shape)
    i = np.arange(n * n).reshape(n, n)
    a, b, c, d = i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, :-1].ravel(), i[1:, 1:].ravel()
    f = np.concatenate([np.stack([a, b, c], 1), np.stack([b, d, c], 1)]).astype(np.int32)
    return v0, v0 + g.normal(0, motion + 1e-300, v0.shape), f


def _triangles(v0, v1):
    f = np.arange(len(v0), dtype=np.int32).reshape(-1, 3)
    return v0, v1, f


def _scene(kind):
    from p2cccd_b200 import scenes

    g = np.random.default_rng(3)
    if kind == "oversized":  # 1,250 small triangles and six that reach across them
        big = g.uniform(0, 1, (18, 3)) * [1.0, 1.0, 0.01]
        objs = [_sheet(26, 0.04, motion=0.01), _triangles(big, big + 0.02)]
    elif kind == "far":  # the rounding guard of the columns is wider than a column
        objs = [tuple(x + 1e6 if x.dtype == np.float64 else x for x in _sheet(12, 1e-7, seed=k, motion=1e-8))
                for k in (0, 1)]
    elif kind == "flat":
        v = np.concatenate([g.uniform(0, 1, (90, 2)), np.zeros((90, 1))], 1)
        objs = [_triangles(v, v.copy())]
    elif kind == "coincident":
        v = np.tile([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]], (60, 1))
        objs = [_triangles(v, v.copy())]
    elif kind == "one":
        v = g.uniform(0, 1, (3, 3))
        objs = [_triangles(v, v + 0.1)]
    elif kind == "three":
        v, f = scenes.uv_sphere(16, 12)
        objs = [(v + [1.9 * k, 0.3 * k, 0], v + [1.8 * k, 0.3 * k, 0.1], f) for k in range(3)]
    else:  # "many": more objects than envelopes are kept for
        objs = []
        for _ in range(70):
            v = g.uniform(0, 0.4, (6, 3)) + g.uniform(0, 1, 3)
            objs.append(_triangles(v, v + g.normal(0, 0.1, 3)))
    return scenes.combine([(a, b, f, scenes.unique_edges(f)) for a, b, f in objs])


def _expected(oracle_mod, s, thickness, exclude_self):
    allowed = oracle_mod.object_allowed(s["v_t0"], s["v_t1"], s["v_obj"], s["n_obj"], thickness, exclude_self)
    box = lambda prim, k: oracle_mod.swept_boxes(s["v_t0"], s["v_t1"], prim, k, thickness)  # noqa: E731
    valid = (s["v_obj"] >= 0).astype(np.uint8)
    vf = oracle_mod.vf_pairs(box(None, 1), s["v_obj"], valid, box(s["faces"], 3), s["f_obj"], s["faces"], allowed,
                             "brute")
    return np.sort(vf), np.sort(oracle_mod.ee_pairs(box(s["edges"], 2), s["e_obj"], s["edges"], allowed, "brute"))


@pytest.mark.parametrize("thickness", [0.0, 1e-3])
@pytest.mark.parametrize("exclude_self", [False, True])
@pytest.mark.parametrize("kind", ["oversized", "far", "flat", "coincident", "one", "three", "many"])
def test_pair_sets(cuda_device, oracle_mod, kind, exclude_self, thickness):
    from p2cccd_b200.scene import ScenePipeline

    s = _scene(kind)
    if kind == "far":
        thickness *= 1e-4
    for cap in (1 << 10, 1 << 16):  # below and above the rank sort's limit
        p = ScenePipeline(s, cuda_device, thickness=thickness, exclude_self=exclude_self, vf_capacity=cap,
                          ee_capacity=cap)
        p.step_checked()
        for got, want in zip(p.pairs(), _expected(oracle_mod, s, thickness, exclude_self)):
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("cap", [8000, 16384, 16385])
def test_rank_sort_limit(cuda_device, oracle_mod, cap):
    """The rank sort's largest buffer, one more entry, and a list that
    overflows its buffer (sorted, members of the set, no repeats)."""
    from p2cccd_b200.scene import ScenePipeline

    s = _scene("oversized")
    p = ScenePipeline(s, cuda_device, exclude_self=False, thickness=0.012, vf_capacity=cap, ee_capacity=cap)
    p.candidates()
    want = _expected(oracle_mod, s, 0.012, False)
    assert p.read_counts() == (len(want[0]), len(want[1]), 0) and 4096 < len(want[0]) < 8000 < len(want[1]) < 16384
    for pairs, w in zip((p.vf_pairs, p.ee_pairs), want):
        got = pairs.cpu().numpy().view(np.uint64)
        if len(w) <= cap:
            np.testing.assert_array_equal(got[:len(w)], w)
            assert (got[len(w):] == np.uint64(2**64 - 1)).all()
        else:
            assert (got[1:] > got[:-1]).all() and np.isin(got, w).all()
