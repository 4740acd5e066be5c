"""Batched any-hit on both sides of the line between selection and full sorts
(K = 4,096): every scene gets what it gets alone."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import anyhit_case as A
from test_batch_anyhit_gpu import _exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top_k", [4096, 4097, 20000])
def test_more_proposals_than_a_block_orders(cuda_device, top_k):
    from p2cccd_b200 import scenes
    from p2cccd_b200.anyhit import BatchAnyHit, GroupAnyHit, stub_scores
    from p2cccd_b200.batch import BatchPipeline
    from p2cccd_b200.certify import CertConfig

    cfg = CertConfig(A.CFG["eps_time"], A.CFG["eps_space"], A.CFG["max_depth"])
    batch = [scenes.cloth_on_sphere(n=65, sphere_lon=40, sphere_rings=30), A.cloth_small(), A.sphere_cluster(7, 5)]
    bp = BatchPipeline(batch, cuda_device, config=cfg, exclude_self=False)
    bp.step_checked()
    counts = bp.read_counts()
    assert max(bp.ee_caps) > 20000 and int(counts[0, 1]) > 20000
    ah = BatchAnyHit(bp.table_host, bp.table, 3, cuda_device, keep_candidates=True)
    seeds = torch.tensor([11, 12, 13], dtype=torch.int64, device=cuda_device)
    ah.run(top_k, cfg, seeds=seeds)
    torch.cuda.synchronize(cuda_device)
    summ = ah.read_summaries()
    for i in range(bp.n):
        for fam, name, caps, off in ((1, "vf", bp.vf_caps, bp.vf_pair_off), (2, "ee", bp.ee_caps, bp.ee_pair_off)):
            pairs = (bp.vf_pairs if fam == 1 else bp.ee_pairs)[int(off[i]):int(off[i]) + caps[i]]
            count = torch.tensor([int(counts[i, fam - 1])], dtype=torch.int64, device=cuda_device)
            scores = torch.empty(caps[i], dtype=torch.float64, device=cuda_device)
            stub_scores(pairs, count, fam, int(seeds[i]), scores)
            one = GroupAnyHit(bp.structs[i], bp.n_obj[i], name, caps[i], cuda_device)
            one.run(pairs, count, scores, top_k, cfg)
            torch.cuda.synchronize(cuda_device)
            assert _exact(summ[i][name]) == _exact(one.read_summary()), (i, name)
            assert np.array_equal(ah.group_detected_of(i, fam), one.read_groups()[0]), (i, name)
            n = int(counts[i, fam - 1])
            for got, want in zip(ah.candidates_of(i, fam, n), one.read_candidates(n)):
                assert np.array_equal(got, want), (i, name)
