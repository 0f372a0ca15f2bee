"""Wells with a barrier up to where f = 1 + T is negative (test_gpu_barrier_levels.py)
where a lane marches each trial energy: batches of 512 and more, the static count
of more than 199 energies."""
from __future__ import annotations

import pytest

import test_gpu_barrier_levels as B

pytestmark = pytest.mark.gpu


def test_lane_scanned_batch(ctx):
    B._check(ctx, [i % len(B._wells()[0]) for i in range(512)], B.FINE)


@pytest.mark.parametrize("n_trial", [200, 1024, 8192])
def test_static_counts_on_lanes(n_trial):
    B._static_check(n_trial)
