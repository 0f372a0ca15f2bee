"""Levels whose window takes a cluster of four CTAs (batches of at most 16
potentials, windows above 16384 points) against a warp per level on the same
batch (epscu_opts.long_window forces it), with the project's bars: energies
within 1e-10 Hartree, node counts exact, wavefunctions within 1e-8 in L2.
Windows around one strip of 16 points per thread (1024 threads), on either side
of the threshold and of the batch size, with the CTA and the warp list filled
beside them; and the wavefunctions the adjoint computes again are the solve's,
so the gradient of a solve that kept them is the same to rounding of its sums."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

WARP = 1 << 24


@pytest.mark.parametrize("B, N", [(1, 16384), (1, 16400), (2, 17000), (3, 32769), (1, 40001), (1, 131071), (2, 150000),
                                  (16, 20001), (17, 20001)])
def test_clusters_match_warps(ctx, B, N):
    b = synth.morse_batch(B=B, N=N, seed=40 + B)
    args = (b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 2048)
    a = ctx.solve(*args, level_capacity=200, want_psi=True)
    c = ctx.solve(*args, level_capacity=200, want_psi=True, long_window=WARP)
    assert np.array_equal(a.n_total, c.n_total)
    assert int(a.n_out.sum()) > 0
    for p in range(B):
        n = int(a.n_out[p])
        assert n == int(c.n_out[p])
        assert np.array_equal(a.nodes[p, :n], np.arange(n)), p
        assert np.max(np.abs(a.energy[p, :n] - c.energy[p, :n])) < 1e-10, p
        h = (np.broadcast_to(b.r_max, B)[p] - np.broadcast_to(b.r_min, B)[p]) / (N - 1)
        err = np.sqrt(np.sum((a.wavefunctions(p) - c.wavefunctions(p)) ** 2, axis=1) * h)
        assert err.max() < 1e-8, (p, int(err.argmax()), err.max())


@pytest.mark.parametrize("B, N", [(1, 16400), (2, 70001)])
def test_recomputed_wavefunctions(ctx, B, N):
    import torch

    b = synth.morse_batch(B=B, N=N, seed=50 + B)
    db = capi.DeviceBatch(ctx, b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 2048, 200, want_psi=True,
                          psi_capacity=200 * B * N)
    db.solve()
    gE = torch.ones(B, 200, dtype=torch.float64, device="cuda")
    db.adjoint(gE)
    kept = db.gV.clone()
    db.adjoint(gE, recompute=True)
    torch.cuda.synchronize()
    scale = float(kept.abs().max())
    assert scale > 0
    assert float((db.gV - kept).abs().max()) <= 1e-13 * scale
