"""Non-finite coordinates are reported and file no box: a vertex, or a whole
face, that is NaN or infinite in one frame or both, with self pairs (nothing
is culled), without, and with more objects than culling handles.  The lists
hold exactly the pairs of the primitives that stay finite, as overlap is a
matter of the two boxes alone."""
from __future__ import annotations

import numpy as np
import pytest

from test_bins_gpu import _expected, _scene, _sheet

pytestmark = pytest.mark.gpu


def _base(kind):
    from p2cccd_b200 import scenes

    if kind != "sheet":
        return _scene(kind)
    v0, v1, f = _sheet(64, 0.02, motion=0.01)
    return scenes.combine([(v0, v1, f, scenes.unique_edges(f))])


def _spoil(s, where, value, frames):
    """A copy with some coordinates replaced, and the vertices they belong to."""
    bad = dict(s, v_t0=s["v_t0"].copy(), v_t1=s["v_t1"].copy())
    n = len(s["v_t0"])
    v, axes = {"vertex": ([n // 2], [0, 1, 2]), "x": ([n // 2], [0]), "z": ([n // 3], [2]),
               "face": (list(s["faces"][len(s["faces"]) // 2]), [0, 1, 2]), "first": ([0], [0, 1, 2]),
               "all": (list(range(n)), [1])}[where]
    for k in frames:
        bad[k][np.ix_(v, axes)] = value
    return bad, np.array(v)


def _without(pairs, s, v):
    """vf and ee keys of the primitives none of whose vertices is in v."""
    vf, ee = pairs
    a, b = vf >> np.uint64(32), vf & np.uint64(0xFFFFFFFF)
    face = np.isin(s["faces"], v).any(axis=1)
    edge = np.isin(s["edges"], v).any(axis=1)
    return (vf[~(np.isin(a, v) | face[b.astype(np.int64)])],
            ee[~(edge[(ee >> np.uint64(32)).astype(np.int64)] | edge[(ee & np.uint64(0xFFFFFFFF)).astype(np.int64)])])


FRAMES = [("v_t0", "v_t1"), ("v_t1",)]


@pytest.mark.parametrize("frames", FRAMES)
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kind,exclude_self", [("sheet", False), ("three", False), ("three", True), ("many", True)])
def test_single_scene(cuda_device, oracle_mod, kind, exclude_self, value, frames):
    from p2cccd_b200.scene import ScenePipeline

    s = _base(kind)
    want = _expected(oracle_mod, s, 1e-3, exclude_self)
    for where in ("vertex", "x", "z", "face", "first", "all"):
        bad, v = _spoil(s, where, value, frames)
        for cap in (1 << 14, 1 << 18):  # both orders of the pair lists
            p = ScenePipeline(bad, cuda_device, thickness=1e-3, exclude_self=exclude_self, vf_capacity=cap,
                              ee_capacity=cap)
            p.candidates()
            finite = _without(want, s, v)
            assert p.read_counts() == (len(finite[0]), len(finite[1]), 1), where
            if max(map(len, finite)) <= cap:
                for got, w in zip(p.pairs(), finite):
                    np.testing.assert_array_equal(got, w)
        with pytest.raises(ValueError, match="finite"):
            p.step_checked()


@pytest.mark.parametrize("frames", FRAMES)
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("exclude_self", [False, True])
def test_batch(cuda_device, oracle_mod, exclude_self, value, frames):
    """Spoiled scenes between whole ones, which keep their lists."""
    from p2cccd_b200.batch import BatchPipeline

    batch, want = [], []
    for kind, where in [("three", None), ("sheet", "vertex"), ("sheet", None), ("sheet", "x"), ("three", "z"),
                        ("sheet", "face"), ("three", "all"), ("three", "first"), ("many", "vertex"), ("three", None)]:
        s = _base(kind)
        w = _expected(oracle_mod, s, 1e-3, exclude_self)
        if where is not None:
            s, v = _spoil(s, where, value, frames)
            w = _without(w, s, v)
        batch.append(s)
        want.append((where is not None, w))
    p = BatchPipeline(batch, cuda_device, thickness=1e-3, exclude_self=exclude_self)
    p._alloc([len(w[0]) + 5 for _, w in want], [len(w[1]) + 5 for _, w in want])
    p.candidates()
    counts = p.read_counts()
    for i, (spoiled, w) in enumerate(want):
        assert tuple(int(x) for x in counts[i, :3]) == (len(w[0]), len(w[1]), int(spoiled)), i
        for got, x in zip(p.pairs(i), w):
            np.testing.assert_array_equal(got, x)
    with pytest.raises(ValueError, match="finite"):
        p.step_checked()


@pytest.mark.parametrize("exclude_self", [False, True])
def test_largest_coordinates(cuda_device, oracle_mod, exclude_self):
    """Finite coordinates whose differences overflow."""
    from p2cccd_b200.batch import BatchPipeline
    from p2cccd_b200.scene import ScenePipeline

    s = dict(_base("three"))
    for k in ("v_t0", "v_t1"):
        s[k] = s[k].copy()
        s[k][::60] *= 8e307 / np.abs(s[k]).max()
        s[k][5] = [1.7e308, -1.7e308, 1.7e308]
        s[k][9] = [-1.7e308, 1.7e308, -1.7e308]
    want = _expected(oracle_mod, s, 0.0, exclude_self)
    p = ScenePipeline(s, cuda_device, exclude_self=exclude_self, vf_capacity=1 << 19, ee_capacity=1 << 19)
    p.candidates()
    b = BatchPipeline([s, _base("three")], cuda_device, exclude_self=exclude_self)
    b._alloc([1 << 19] * 2, [1 << 19] * 2)
    b.candidates()
    assert p.read_counts() == (len(want[0]), len(want[1]), 0) == tuple(int(x) for x in b.read_counts()[0, :3])
    for got, one, w in zip(p.pairs(), b.pairs(0), want):
        np.testing.assert_array_equal(got, w)
        np.testing.assert_array_equal(one, w)
