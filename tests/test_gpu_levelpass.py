"""The group passes of the fast method at the sizes where they can go wrong:
grids of a few points, windows around one strip (16 points), one warp's strips
(512) and one CTA's (4096), on a warp and on a CTA per level
(epscu_opts.long_window forces either), double wells whose levels pair up, and
a barrier above the cut-offs inside the grid.  Against the plain FP64 method
(bit-exact with the oracle), with the project's bars: energies within 1e-10
Hartree, node counts exact, wavefunctions within 1e-8 in L2."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

WARP, CTA = 1 << 24, 1


def _check(ctx, V, r0, r1, mu, cap, n_trial, long_window, psi_tol=1e-8):
    args = (V, r0, r1, mu, cap, n_trial)
    ref = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=160, want_psi=True)
    sol = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=160, want_psi=True, long_window=long_window)
    assert np.array_equal(sol.n_total, ref.n_total)
    levels = 0
    for p in range(len(V)):
        n = int(ref.n_out[p])
        assert int(sol.n_out[p]) == n
        if n == 0 or ref.status[p, 0] & capi.LEVEL_UNDER_RESOLVED:
            continue
        levels += n
        assert np.max(np.abs(sol.energy[p, :n] - ref.energy[p, :n])) < 1e-10, p
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), p
        assert np.all(sol.status[p, :n] == 0)
        h = (np.broadcast_to(r1, len(V))[p] - np.broadcast_to(r0, len(V))[p]) / (V[p].size - 1)
        err = np.sqrt(np.sum((sol.wavefunctions(p) - ref.wavefunctions(p)) ** 2, axis=1) * h)
        assert err.max() < psi_tol, (p, int(err.argmax()), err.max())
    return levels


@pytest.mark.parametrize("long_window", [WARP, CTA])
def test_tiny_grids(ctx, long_window):
    """5 to 70 points over a harmonic well: sides shorter than a strip, with
    the window's ends at the cut-offs."""
    sizes = [5, 6, 7, 8, 15, 16, 17, 18, 31, 32, 33, 34, 35, 47, 48, 49, 63, 64, 65, 70]
    V, mu = [], []
    for N in sizes:
        r = np.linspace(-1.0, 1.0, N)
        h = r[1] - r[0]
        V.append(0.5 * r * r)
        mu.append(0.4 / (2.0 * 0.499 * h * h) * 0.5)  # k_max h < 1
    n = _check(ctx, V, -1.0, 1.0, np.array(mu), 0.499, 64, long_window)
    assert n > 20


@pytest.mark.parametrize("long_window", [WARP, CTA])
@pytest.mark.parametrize("N", [511, 512, 513, 529, 4095, 4097, 8193, 16411])
def test_window_edges(ctx, N, long_window):
    """Morse wells whose windows end in the grid and at its ends, across the
    sizes where a thread's strip count changes."""
    De, a, re = 0.1, 1.0, 2.0
    V, r1 = [], np.array([re + 4.0, re + 9.0, re + 30.0])
    for b in r1:
        V.append(synth.morse(np.linspace(0.5, b, N), De, a, re))
    h = (r1[-1] - 0.5) / (N - 1)
    mu = min(20000.0, 0.8 / (2 * De * h * h))
    assert _check(ctx, V, 0.5, r1, mu, 0.999 * De, 1024, long_window) >= 3


@pytest.mark.parametrize("long_window", [WARP, CTA])
def test_paired_levels_of_double_wells(ctx, long_window):
    """Symmetric and slightly tilted double wells: pairs split by less than the
    scan's spacing, down to 1e-9 Hartree, which the FP32 stage cannot tell
    apart.  (A pair mixes freely within its splitting: psi is compared
    where the splitting is wide against the energy's resolution.)"""
    r = np.linspace(-2.5, 2.5, 3001)
    V = [0.05 * (r * r - 1.0) ** 2 + tilt * r for tilt in (0.0, 1e-6, 1e-3)]
    compared = 0
    for n_trial in (512, 16):
        args = (V, -2.5, 2.5, 2000.0, 0.04, n_trial)
        ref = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=64, want_psi=True)
        sol = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=64, want_psi=True, long_window=long_window)
        assert np.array_equal(sol.n_total, ref.n_total)
        for p in range(len(V)):
            n = int(ref.n_out[p])
            assert n > 4 and int(sol.n_out[p]) == n
            E = ref.energy[p, :n]
            assert np.max(np.abs(sol.energy[p, :n] - E)) < 1e-10
            assert np.array_equal(sol.nodes[p, :n], np.arange(n))
            gap = np.array([np.min(np.abs(np.delete(E, v) - E[v])) for v in range(n)])
            err = np.sqrt(np.sum((sol.wavefunctions(p) - ref.wavefunctions(p)) ** 2, axis=1) * (r[1] - r[0]))
            wide = gap > 1e-4
            assert np.all(err[wide] < 1e-8)
            compared += int(wide.sum())
    assert compared > 4


@pytest.mark.parametrize("long_window", [WARP, CTA])
def test_barrier_above_the_cut_offs(ctx, long_window):
    """A barrier inside the grid with a (V - V_min) up to 0.9 (1 + T down to
    0.1): the solution grows ~100-fold a point there."""
    r = np.linspace(0.0, 4.0, 801)
    h = r[1] - r[0]
    mu = 4000.0
    a = mu * h * h / 6.0
    V = [0.05 * (r - 1.0) ** 2 + top / a * np.exp(-((r - 2.5) ** 2) / (2 * 0.04 ** 2)) for top in (0.45, 0.6, 0.9)]
    assert max(v[400:600].max() for v in V) * a > 0.8
    assert _check(ctx, V, 0.0, 4.0, mu, 0.04, 512, long_window) >= 9
