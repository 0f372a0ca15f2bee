"""Levels of such wells that share a scan bracket, or nearly."""
from __future__ import annotations

import pytest

import test_gpu_barrier_levels as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_trial", [1, 16, 64, 512])
@pytest.mark.parametrize("batch", [40, 512])
def test_levels_that_share_a_bracket(ctx, batch, n_trial):
    B._check(ctx, [i % len(B._wells()[0]) for i in range(batch)], n_trial)
