"""Workspace sizes over the whole range of counts an entry point accepts: each
call returns (a child process with a time limit, so that one that never does
is a failure), and sizes grow with the count."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

CODE = """
import sys
sys.path.insert(0, {pkg!r})
from p2cccd_b200 import _lib
size = _lib.load().p2c_proposal_feature_rows_workspace_bytes
print(*[size(n) for n in {counts}])
"""


def test_feature_row_workspace_of_every_proxy_count():
    counts = [0, 1, 1000, 1 << 20, (1 << 29) + 3, 1 << 30, (1 << 30) + 1, 3 << 29, (1 << 31) - 1]
    out = subprocess.run([sys.executable, "-c", CODE.format(pkg=str(ROOT / "p2c-ccd_b200"), counts=counts)],
                         capture_output=True, text=True, timeout=120, check=True).stdout
    sizes = [int(x) for x in out.split()]
    assert len(sizes) == len(counts) and sizes == sorted(sizes)
    assert all(44 * n <= size <= 80 * n + (1 << 20) for n, size in zip(counts, sizes))
