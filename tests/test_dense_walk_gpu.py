"""The walk of a candidate group at the lengths where its look-ahead changes:
three steps of 32 rows are on their way while one is worked on.  Totals are
compared bit for bit."""
from __future__ import annotations

import pytest

from test_dense_groups import _same
from test_dense_order_gpu import _sized_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [{"threshold": 0.97, "limit": 40}, {"preserve": True}, {"threshold": 0.999, "limit": 100000}])
def test_walk_of_every_length(cuda_device, oracle_mod, cfg):
    from p2cccd_b200.dense_groups import DenseGroupEarlyStop, _query_bits, upload

    edges = [32 * k + d for k in range(1, 9) for d in (-1, 0, 1)]
    for sizes in ([n] for n in edges):
        rows = _sized_rows(sizes, 5)
        _check(cuda_device, oracle_mod, rows, cfg, DenseGroupEarlyStop, _query_bits, upload)
    _check(cuda_device, oracle_mod, _sized_rows(edges * 20 + [1, 2, 3] * 50, 6), cfg, DenseGroupEarlyStop, _query_bits,
           upload)


def _check(device, oracle_mod, rows, cfg, runner, bits, upload):
    n = len(rows["query_id"])
    r = runner(n, device)
    r.run(upload(rows, device), n, query_bits=bits(rows["query_id"]), **cfg)
    assert _same(r.result(), oracle_mod.dense_group(rows, **cfg)) == []
