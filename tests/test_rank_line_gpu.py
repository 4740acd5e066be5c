"""Both sides of the line between pair lists ordered by rank and by rows."""
from __future__ import annotations

import pytest

import test_bins_gpu as bins

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [8191, 8192, 8193, 12000])
def test_orders_agree_with_the_oracle(cuda_device, oracle_mod, cap):
    bins.test_rank_sort_limit(cuda_device, oracle_mod, cap)
