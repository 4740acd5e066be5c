"""The warp engine at the sizes where its groups, batches and stack change
shape, byte for byte against the CPU oracle (no tolerance).

* 1, 3, 6 and 10 queries are the largest batches whose roots are sampled with
  four, three, two and one level per group; one more query changes the shape.
* Grazing queries whose trees are full to a given depth fill the warp's stack
  (256 nodes, of which 64 stay free) and the pool other warps take from.
* Leaves right of a collision, sampled by speculation, must not count."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bytes(a):
    return np.ascontiguousarray(a).view(np.uint8).reshape(-1, 72)


def _check(oracle_mod, rec, fam, interval, cfg):
    import torch
    from p2cccd_b200 import certify

    out = certify.certify_batch(certify.records_to_device(rec), fam, *interval, certify.CertConfig(*cfg))
    torch.cuda.synchronize()
    cpu, st, _ = oracle_mod.eval_batch(rec, *interval, *cfg)
    assert st.sum() == 0
    np.testing.assert_array_equal(_bytes(certify.results_to_numpy(out)), _bytes(cpu))


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 7, 10, 11, 33])
@pytest.mark.parametrize("interval", [(0.0, 1.0), (0.1, 0.7)])
def test_small_batches(cuda_device, oracle_mod, n, interval):
    from p2cccd_b200 import workloads

    w = workloads.plain_queries(workloads.PlainSpec(n_vf=n, n_ee=n, seed=100 + n, touch_frac=0.6))
    for fam, name in ((1, "vf"), (2, "ee")):
        _check(oracle_mod, w[name], fam, interval, (1e-6, 1e-6, 32))


def _grazing(n: int, span: float, lift: float):
    """Points sliding by ``span`` over a fixed triangle at eps_space + lift:
    every interval wider than about 2 lift / span stays undecided, so the
    trees are full down to that depth (or to the depth limit)."""
    from p2cccd_b200 import records

    g = np.random.default_rng(n)
    p0 = np.zeros((n, 4, 3))
    p0[:, 1:, :] = [[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]]
    p1 = p0.copy()
    p0[:, 0, :] = np.stack([g.uniform(0.05, 0.2, n), g.uniform(0.05, 0.2, n), np.full(n, 1e-6 + lift)], 1)
    p1[:, 0, :] = p0[:, 0, :] + [span, 0.0, 0.0]
    return records.pack_primitives(p0, p1, np.arange(n), np.arange(n) + 10)


@pytest.mark.parametrize("n,depth", [(1, 10), (1, 16), (5, 14), (700, 11)])
def test_full_trees(cuda_device, oracle_mod, n, depth):
    _check(oracle_mod, _grazing(n, 0.3, 1e-9), 1, (0.0, 1.0), (1e-12, 1e-6, depth))  # undecided at the limit
    _check(oracle_mod, _grazing(n, 0.3, 0.3 / 2 ** depth), 1, (0.0, 1.0), (1e-12, 1e-6, 40))  # separated there


@pytest.mark.parametrize("toi", [0.03, 0.4999, 0.51, 0.97])
def test_first_hit_wins(cuda_device, oracle_mod, toi):
    """A point that crosses the triangle at ``toi``."""
    from p2cccd_b200 import records

    n = 64
    g = np.random.default_rng(7)
    p0 = np.zeros((n, 4, 3))
    p0[:, 1:, :] = [[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]]
    p1 = p0.copy()
    z = g.uniform(0.1, 1.0, n)
    p0[:, 0, :] = np.stack([g.uniform(0.1, 0.4, n), g.uniform(0.1, 0.4, n), z], 1)
    p1[:, 0, :] = p0[:, 0, :]
    p1[:, 0, 2] = z * (1.0 - 1.0 / toi)
    rec = records.pack_primitives(p0, p1, np.arange(n), np.arange(n) + 10)
    _check(oracle_mod, rec, 1, (0.0, 1.0), (1e-6, 1e-6, 32))
