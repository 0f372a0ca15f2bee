"""Levels the refinement hands over to the repair kernel: wells with bumps,
where a level's match point can lie in another well than the level and the pass
there never shows the level's node count (the kernel halves the bracket a few
times, then looks for a better point).  Against the plain FP64 method, with the
project's bars: energies within 1e-10 Hartree, node counts exact, wavefunctions
within 1e-8 in L2 (levels at least 1e-6 Hartree from the next)."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

WARP, CTA = 1 << 24, 1


@pytest.mark.parametrize("long_window", [WARP, CTA])
def test_bumped_wells(ctx, long_window):
    b = synth.bump_adjoint(B=160, N=4096, n_trial=1024, seed=4, amp_scale=4.0)
    b = b[0] if isinstance(b, tuple) else b
    args = (b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 1024)
    # (energies to the last bits: a wavefunction's error is the energy's over the
    # gap to the next level, 2e-8 at gaps of 3e-5 with brackets of 1e-12)
    ref = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=200, want_psi=True, tol=1e-15)
    sol = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=200, want_psi=True, long_window=long_window)
    handed_over = ctx.stats().fallbacks
    assert np.array_equal(sol.n_total, ref.n_total)
    for p in range(160):
        n = int(ref.n_out[p])
        if n < 2 or ref.status[p, 0] & capi.LEVEL_UNDER_RESOLVED:
            continue
        E = ref.energy[p, :n]
        assert np.max(np.abs(sol.energy[p, :n] - E)) < 1e-10, p
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), p
        gap = np.minimum(np.diff(E, prepend=-1.0), np.diff(E, append=1e9))
        h = (np.broadcast_to(b.r_max, 160)[p] - np.broadcast_to(b.r_min, 160)[p]) / 4095
        err = np.sqrt(np.sum((sol.wavefunctions(p) - ref.wavefunctions(p)) ** 2, axis=1) * h)
        assert np.all(err[gap > 1e-6] < 1e-8), p
    assert handed_over > 0
