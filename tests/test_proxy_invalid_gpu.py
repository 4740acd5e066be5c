"""Proxies whose bounds have no order or are not finite are reported (error
bit 1) whatever the width hints: with a direct slab table, without one, and
without hints.  The hits between the other proxies are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HINTS = [(2, 3, 7), (6, 3, 7), (7, 3, 7), (20, 20, 20), (0, 0, 0)]


def _spoil(bounds, how):
    """Rows of (min xyz, max xyz), in place."""
    if how.startswith("reversed"):
        for a in map(int, how.split("_")[1]):
            bounds[:, [a, 3 + a]] = bounds[:, [3 + a, a]]
    elif how.startswith("far"):  # reversed across every other proxy
        a = int(how.split("_")[1])
        bounds[:, a], bounds[:, 3 + a] = 5.0, -5.0
    else:
        value, cols = how.split("_")
        bounds[:, list(map(int, cols))] = float(value)


@pytest.mark.parametrize("how", ["reversed_0", "reversed_1", "reversed_2", "reversed_01", "reversed_12", "reversed_012",
                                 "far_0", "far_1", "far_2", "nan_0", "nan_3", "nan_5", "nan_012345", "inf_3", "inf_0",
                                 "-inf_1", "-inf_5", "inf_012345"])
@pytest.mark.parametrize("hint", HINTS)
def test_invalid_bounds(cuda_device, oracle_mod, how, hint):
    from p2cccd_b200 import scenes
    from p2cccd_b200.proxy import ProxyCandidates, RAW_HIT_DTYPE

    sc = scenes.proxy_scene(n_objects=6, patches_per_object=60, n_slabs=3, seed=12)
    ref_raw, _ = oracle_mod.proxy_candidates(sc)
    assert len(ref_raw) > 500
    for count in (1, 40):
        bad = np.random.default_rng(count).choice(sc["n"], count, replace=False)
        bounds = sc["bounds"].copy()
        rows = bounds[bad]
        _spoil(rows, how)
        bounds[bad] = rows
        pc = ProxyCandidates(dict(sc, bounds=bounds, id_bits=hint), cuda_device, raw_capacity=1 << 19)
        pc.run()
        n_raw, _, err = (int(x) for x in pc.counts[:3].cpu())
        assert err & 1 and n_raw <= pc.cap
        raw = pc.raw[:n_raw].cpu().numpy().view(RAW_HIT_DTYPE).reshape(-1)
        clean = lambda r: r[~(np.isin(r["proxy_a_index"], bad) | np.isin(r["proxy_b_index"], bad))]  # noqa: E731
        assert clean(raw).tobytes() == clean(ref_raw).tobytes()
        with pytest.raises(ValueError, match="finite ordered bounds"):
            pc.run_checked()
