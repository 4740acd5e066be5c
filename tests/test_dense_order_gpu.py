"""The order inside candidate groups at the sizes where its path changes (a
warp's 256 rows, a block's tile of 4,096, one merge, several), and the ordered
totals over many pieces.  Totals are compared bit for bit: they are sums whose
order the reference fixes."""
from __future__ import annotations

import numpy as np
import pytest

from dense_inputs import make_rows
from test_dense_groups import _same

pytestmark = pytest.mark.gpu


def _sized_rows(sizes, seed):
    rows = make_rows(sum(sizes), seed)
    rng = np.random.default_rng(seed)
    rows["query_id"] = rng.permutation(np.repeat(np.arange(1, len(sizes) + 1, dtype=np.uint64), sizes))
    return rows


@pytest.mark.parametrize("sizes", [[1], [2, 1, 31, 32, 33], [255, 256, 257, 3], [4095, 4096, 4097, 1],
                                   [8191, 8192, 8193, 40, 12289], [60001, 5000, 300, 2], [1] * 3000 + [4097]])
@pytest.mark.parametrize("cfg", [{"threshold": 0.97, "limit": 40}, {"preserve": True},
                                 {"threshold": 0.999, "limit": 100000, "penalty": 0.0}])
def test_order_inside_groups(cuda_device, oracle_mod, sizes, cfg):
    from p2cccd_b200.dense_groups import DenseGroupEarlyStop, _query_bits, upload

    rows = _sized_rows(sizes, 21)
    n = len(rows["query_id"])
    r = DenseGroupEarlyStop(n, cuda_device)
    r.run(upload(rows, cuda_device), n, query_bits=_query_bits(rows["query_id"]), **cfg)
    assert _same(r.result(), oracle_mod.dense_group(rows, **cfg)) == []


@pytest.mark.parametrize("scale", ["even", "wide", "grows", "huge"])
def test_totals_over_many_pieces(cuda_device, oracle_mod, scale):
    """150,000 rows: the totals run over dozens of 4,096-term pieces; costs of
    every magnitude, costs that grow along the sequence (a binade step in most
    pieces) and a sum that overflows."""
    from p2cccd_b200.dense_groups import DenseGroupEarlyStop, _query_bits, upload

    n = 150000
    rows = make_rows(n, 33)
    rng = np.random.default_rng(34)
    full = rows["oracle_trace"][:, 5]
    if scale == "wide":
        full[:] = np.exp(rng.uniform(-60.0, 60.0, n))
    elif scale == "grows":
        full[:] = np.exp2(rows["query_id"].astype(np.float64) * (60.0 / rows["query_id"].max()))
    elif scale == "huge":
        full[:] = 1e303 * rng.random(n)
    r = DenseGroupEarlyStop(n, cuda_device)
    r.run(upload(rows, cuda_device), n, query_bits=_query_bits(rows["query_id"]))
    assert _same(r.result(), oracle_mod.dense_group(rows)) == []
