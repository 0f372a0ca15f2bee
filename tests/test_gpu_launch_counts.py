"""epscu_stats.kernel_launches: the kernels of each pipeline (the plain method with
and without wavefunctions, the fast one with the lane and the group scan)."""
from __future__ import annotations

import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B, method, psi, launches", [
    (3, capi.METHOD_PLAIN_FP64, False, 10),
    (3, capi.METHOD_PLAIN_FP64, True, 11),
    (3, capi.METHOD_FAST_FP32C, True, 16),
    (512, capi.METHOD_FAST_FP32C, False, 15),
])
def test_launches(ctx, B, method, psi, launches):
    b = synth.morse_batch(B=B, N=1000, seed=4)
    ctx.solve(b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 256, method=method, level_capacity=64, want_psi=psi)
    assert ctx.stats().kernel_launches == launches
