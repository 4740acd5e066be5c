"""Every way the id width hints can go (keys and lookups by id tables, by packed
words, by ranks, without hints) gives the oracle's candidates and one set of
feature rows: records and rows are compared byte for byte."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# slab, object, patch bits: tables; one bit past the group table; packed words with rank keys;
# too wide for a packed word; none
HINTS = [(3, 3, 7), (3, 12, 7), (6, 12, 20), (20, 20, 20), (0, 0, 0)]


@pytest.mark.parametrize("slabs,objs,patches,dups", [(1, 2, 1, 0.0), (1, 7, 100, 0.3), (5, 8, 33, 0.0), (8, 3, 128, 0.6)])
def test_hints_do_not_change_results(cuda_device, oracle_mod, slabs, objs, patches, dups):
    from p2cccd_b200 import scenes
    from p2cccd_b200.proxy import ProxyCandidates

    sc = scenes.proxy_scene(n_objects=objs, patches_per_object=patches, n_slabs=slabs, seed=41, duplicates=dups)
    if patches == 100:  # all patches in a few columns: windows longer than a whole run
        half = sc["bounds"].reshape(-1, 2, 3)
        half[:, :, 1:] *= 1e-3
    ref_raw, ref_cand = oracle_mod.proxy_candidates(sc)
    first = None
    for hint in HINTS:
        pc = ProxyCandidates(dict(sc, id_bits=hint), cuda_device)
        raw, cand = pc.run_checked()
        assert pc._struct.object_bits == hint[1]  # the hint held
        assert raw.tobytes() == ref_raw.tobytes() and cand.tobytes() == ref_cand.tobytes(), hint
        if len(raw):
            assert pc.compact(raw[::-1].copy()).tobytes() == ref_cand.tobytes(), hint
        dens, rows = pc.feature_rows()
        got = dens.tobytes(), rows.tobytes()
        first = first or got
        assert got == first, hint
        assert len(rows) == len(cand)
