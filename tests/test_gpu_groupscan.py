"""The scan of small batches (a group of threads per trial energy) against the
lane scan of every trial energy, which a batch takes when it sets wait_polls:
level totals and node counts equal, energies of both within the project's bar
of 1e-10 Hartree (the scan gives brackets and first energies only), and
everything of an under-resolved potential equal to the last bit, since it takes
the lane scan either way.  Trial ladders around the coarse stride (16), grids
around one strip per lane (512 points) and on either side of the line where an
energy takes a whole CTA (65536 points), and a batch on either side of the
bisection scan's line (512).  The static count on either side of the line where
it turns from a warp to a lane per energy: the levels below each trial energy,
except within 1e-8 Hartree of a level, where FP32 counts may fall on either
side."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

LANES = 1 << 22  # the default bound of the waits


def _same(ctx, V, r0, r1, mu, cap, n_trial):
    args = (V, r0, r1, mu, cap, n_trial)
    a = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=300)
    c = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=300, wait_polls=LANES)
    assert np.array_equal(a.n_total, c.n_total)
    assert np.array_equal(a.n_out, c.n_out)
    levels = under = 0
    for p in range(len(V)):
        n = int(a.n_out[p])
        levels += n
        if n == 0:
            continue
        assert np.array_equal(a.nodes[p, :n], c.nodes[p, :n]), p
        if a.status[p, 0] & capi.LEVEL_UNDER_RESOLVED:
            under += n
            assert np.array_equal(a.energy[p, :n], c.energy[p, :n]), p
        assert np.max(np.abs(a.energy[p, :n] - c.energy[p, :n])) < 1e-10, p
    return levels, under


@pytest.mark.parametrize("n_trial", [1, 2, 15, 16, 17, 31, 32, 33, 255, 1000])
def test_trial_ladders(ctx, n_trial):
    b = synth.morse_batch(B=5, N=3000, seed=8)
    levels, _ = _same(ctx, b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, n_trial)
    assert levels > 0


def test_grid_edges(ctx):
    sizes = [5, 6, 17, 31, 32, 33, 511, 512, 513, 514, 528, 4096, 4097]
    V = [0.5 * np.linspace(-1.0, 1.0, N) ** 2 for N in sizes]
    mu = np.array([2.0 / (2.0 / (N - 1)) for N in sizes])
    _same(ctx, V, -1.0, 1.0, mu, 0.45, 200)


@pytest.mark.parametrize("B", [1, 3, 60, 511, 512])
def test_batches(ctx, B):
    """every kind, under-resolved potentials among them"""
    b = synth.mixed_batch(B=B, n_min=1024, n_max=9000, n_trial=512, seed=30 + B)
    levels, under = _same(ctx, b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 512)
    assert levels > 0
    assert B < 60 or under > 0


@pytest.mark.parametrize("N", [65535, 65536, 65537, 100003])
def test_long_grids(ctx, N):
    b = synth.morse_batch(B=2, N=N, seed=9)
    levels, _ = _same(ctx, b.potentials(), b.r_min, b.r_max, b.mu, b.e_cap, 700)
    assert levels > 0


@pytest.mark.parametrize("N, n_trial", [(2048, 1), (2500, 2375), (2500, 2376), (10007, 5430), (10007, 5431), (10007, 8192),
                                        (65536, 300)])
def test_static_counts_either_side_of_the_line(ctx, N, n_trial):
    import ctypes as C

    import torch

    b = synth.morse_batch(B=1, N=N, seed=60)
    V = np.ascontiguousarray(b.V(0))
    args = (float(b.r_min[0]), float(b.r_max[0]), float(b.mu[0]), float(b.e_cap[0]))
    sol = ctx.solve([V], *args, 2048, method=capi.METHOD_FAST_FP32C, level_capacity=300)
    E = sol.energy[0, : int(sol.n_out[0])]
    e_lo = V.min()
    Ej = e_lo + (np.arange(n_trial) + 1) * ((args[3] - e_lo) / n_trial)
    near = np.min(np.abs(Ej[:, None] - E[None, :]), axis=1) < 1e-8
    Vd = torch.from_numpy(V).cuda()
    counts = torch.full((n_trial,), -1, dtype=torch.int32, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = capi.load().epscu_count_levels_static(C.cast(C.c_void_p(Vd.data_ptr()), capi._dp), N, *args, n_trial,
                                               C.cast(C.c_void_p(counts.data_ptr()), capi._ip), stream)
    assert rc == 0
    assert E.size > 0
    assert np.array_equal(counts.cpu().numpy()[~near], np.searchsorted(E, Ej)[~near])
