"""Without the reference's libraries a comparison with them is a skip; any
other missing file stays a failure."""
from __future__ import annotations

import conftest
import pytest


def test_missing_reference_library_is_a_skip(oracle_mod, monkeypatch, tmp_path):
    import numpy as np

    monkeypatch.setattr(oracle_mod, "REF_SO", tmp_path / "absent.so")
    monkeypatch.setattr(oracle_mod, "_ref", None)
    with pytest.raises(oracle_mod.ReferenceNotBuilt):
        oracle_mod.ref_eval_batch(np.zeros(1, oracle_mod.PT))
    for error, outcome in ((oracle_mod.ReferenceNotBuilt("absent"), pytest.skip.Exception),
                           (FileNotFoundError("other"), FileNotFoundError)):
        call = conftest.pytest_runtest_call(None)
        next(call)
        with pytest.raises(outcome):
            call.throw(error)
