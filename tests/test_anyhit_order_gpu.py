"""The proposals of a group are its K best candidates by (score desc, index):
tied scores, wide score ranges, groups larger than one block sorts, and K on
both sides of the line between selection and full sorts.

A candidate's recorded phase is a whole number fixed by the procedure, so the
comparison is exact."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import anyhit_case as A

pytestmark = pytest.mark.gpu

PAIRS = 30000


@pytest.fixture(scope="module")
def case(oracle_mod):
    """Random vertex-face pairs of seven spheres, sorted, with their groups and
    certified decisions: most groups hold thousands and few pairs collide."""
    s = A.sphere_cluster(7, 5)
    rng = np.random.default_rng(17)
    nv, nf = len(s["v_t0"]), len(s["faces"])
    keys = np.unique(rng.integers(0, nv, 3 * PAIRS) * nf + rng.integers(0, nf, 3 * PAIRS))
    small = np.nonzero(rng.random(len(keys)) < PAIRS / len(keys))[0]
    cands = np.stack([keys[small] // nf, keys[small] % nf], 1)
    same = (s["faces"][cands[:, 1]] == cands[:, :1]).any(axis=1)
    cands = cands[~same]
    oa, ob = s["v_obj"][cands[:, 0]], s["f_obj"][cands[:, 1]]
    n_obj = int(s["n_obj"])
    groups = (np.minimum(oa, ob) * n_obj + np.maximum(oa, ob)).astype(np.int32)
    return s, cands, groups, n_obj, A.hits(oracle_mod, s, s["edges"], cands, "vf")


def _phases(groups, scores, hit, k):
    out = np.zeros(len(groups), np.uint8)
    for g in np.unique(groups):
        members = np.nonzero(groups == g)[0]
        order = members[np.lexsort((members, -scores[members]))]
        top = order[:k]
        h = np.nonzero(hit[top])[0]
        if len(h):
            out[top[:h[0] + 1]] = 1
            continue
        out[top] = 1
        rest = np.sort(order[k:])
        h = np.nonzero(hit[rest])[0]
        out[rest[:h[0] + 1] if len(h) else rest] = 2
    return out


def _scores(mode, n):
    rng = np.random.default_rng(5)
    if mode == "uniform":
        return rng.random(n)
    if mode == "constant":
        return np.full(n, 0.25)
    if mode == "three_values":
        return rng.integers(0, 3, n).astype(np.float64)
    x = rng.normal(size=n) * 10.0 ** rng.integers(-300, 300, n)  # every exponent, both signs
    x[rng.random(n) < 0.05] = np.inf
    x[rng.random(n) < 0.05] = -np.inf
    x[rng.random(n) < 0.05] = -0.0
    x[rng.random(n) < 0.05] = 5e-324
    return x


@pytest.mark.parametrize("mode", ["uniform", "constant", "three_values", "wide"])
@pytest.mark.parametrize("one_group", [False, True])
def test_proposals_are_the_best_of_each_group(cuda_device, case, mode, one_group):
    from p2cccd_b200.anyhit import GroupAnyHit
    from p2cccd_b200.certify import CertConfig
    from p2cccd_b200.scene import ScenePipeline

    s, cands, groups, n_obj, hit = case
    s = dict(s)
    if one_group:  # 30,000 candidates in the group of object 0 with itself
        s.update(v_obj=np.zeros_like(s["v_obj"]), f_obj=np.zeros_like(s["f_obj"]))
        groups = np.zeros_like(groups)
    pipe = ScenePipeline(s, cuda_device, exclude_self=False)
    n, cap = len(cands), len(cands) + 777
    keys = np.zeros(cap, np.int64)
    keys[:n] = (cands[:, 0].astype(np.int64) << 32) | cands[:, 1]
    scores = np.zeros(cap)
    scores[:n] = _scores(mode, n)
    ah = GroupAnyHit(pipe._struct, n_obj, "vf", cap, cuda_device)
    cfg = CertConfig(A.CFG["eps_time"], A.CFG["eps_space"], A.CFG["max_depth"])
    args = (torch.from_numpy(keys).to(cuda_device), torch.tensor([n], dtype=torch.int64, device=cuda_device),
            torch.from_numpy(scores).to(cuda_device))
    for k in (1, 31, 1024, 4095, 4096, 4097):
        ah.run(*args, k, cfg)
        torch.cuda.synchronize(cuda_device)
        assert ah.read_summary()["error_word"] == 0
        phase, _ = ah.read_candidates(n)
        assert np.array_equal(phase, _phases(groups, scores[:n], hit, k)), k
