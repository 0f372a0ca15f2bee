"""The fast method on wells with a barrier inside the grid, up to where f = 1 + T
is negative and the sign changes of u = f psi number the levels plus the points
with f < 0.  Against the dense solution of the same discrete problem (the
oracle's counts, and with them its energies, are off where a solution has a node
beside such a barrier) and, on grids too long for it, against Sturm counts in
FP64 either side of each level.  The project's bars: energies within 1e-10
Hartree, node counts exact, wavefunctions within 1e-8 in L2 (gaps of 2.7e-4 and
up; the sign is the inner wall's, where some levels are below rounding)."""
from __future__ import annotations

import ctypes as C
import functools

import numpy as np
import pytest

import barrier_wells as W
from epseon_backend_gb300 import capi

pytestmark = pytest.mark.gpu

WARP, CTA = 1 << 24, 1
FINE = 4096  # trial energies closer than any two levels


@functools.cache
def _wells():
    wells = [w[0] for w in W.wells()]
    return wells, [W.dense(V, 1.0, 1.0, W.CAP) for V in wells]


def _check(ctx, which, n_trial, long_window=0):
    wells, refs = _wells()
    sol = ctx.solve([wells[i] for i in which], 0.0, 160.0, 1.0, W.CAP, n_trial, level_capacity=32, want_psi=True,
                    long_window=long_window)
    for p, i in enumerate(which):
        E, psi = refs[i]
        n = int(sol.n_out[p])
        assert int(sol.n_total[p]) == E.size and n == E.size, i
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), i
        assert np.all(sol.status[p, :n] == 0), i
        assert np.max(np.abs(sol.energy[p, :n] - E)) < 1e-10, i
        got = sol.wavefunctions(p)
        err = np.minimum(np.linalg.norm(got - psi, axis=1), np.linalg.norm(got + psi, axis=1))
        assert err.max() < 1e-8, (i, int(err.argmax()), err.max())


@pytest.mark.parametrize("long_window", [WARP, CTA])
def test_batch(ctx, long_window):
    _check(ctx, range(len(_wells()[0])), FINE, long_window)


def test_one_at_a_time(ctx):
    for i in range(len(_wells()[0])):
        _check(ctx, [i], FINE)


def test_largest_group_scanned_batch(ctx):
    _check(ctx, [i % len(_wells()[0]) for i in range(511)], FINE)


def _static(V, r_max, mu, cap, n_trial):
    import torch

    Vd = torch.from_numpy(V).cuda()
    counts = torch.full((n_trial,), -7, dtype=torch.int32, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = capi.load().epscu_count_levels_static(C.cast(C.c_void_p(Vd.data_ptr()), capi._dp), V.size, 0.0, r_max, mu, cap,
                                               n_trial, C.cast(C.c_void_p(counts.data_ptr()), capi._ip), stream)
    assert rc == 0
    return counts.cpu().numpy()


def _static_check(n_trial):
    """(a warp per trial energy up to 9500 N / (7500 + N), 199 here, a lane above;
    within 1e-8 of a level FP32 counts may fall on either side)"""
    for V, (E, _) in zip(*_wells()):
        c = _static(V, 160.0, 1.0, W.CAP, n_trial)
        Ej = V.min() + (np.arange(n_trial) + 1) * ((W.CAP - V.min()) / n_trial)
        near = np.min(np.abs(Ej[:, None] - E[None, :]), axis=1) < 1e-8
        assert np.array_equal(c[~near], np.searchsorted(E, Ej)[~near])


def test_static_counts_on_warps():
    _static_check(199)


@pytest.mark.parametrize("f", W.F_BARRIER)
@pytest.mark.parametrize("N, batch, points", [(20001, 1, 1), (20001, 3, 20), (70001, 1, 3)])
def test_long_grids(ctx, N, batch, points, f):
    """levels of clusters of CTAs, of CTAs and of warps; a CTA per trial energy on
    the longest.  A harmonic well of ~20 levels with the barrier off its centre."""
    mu, omega, cap = 2000.0, 1e-3, 0.02
    r = np.linspace(0.0, 12.0, N)
    h = 12.0 / (N - 1)
    Vs = []
    for q in range(batch):
        V = 0.5 * mu * omega ** 2 * (r - 6.1) ** 2
        at = int((0.42 + 0.05 * q) * N)
        V[at:at + points] = 0.5 * cap + (1.0 - f) / (mu * h * h / 6.0)
        Vs.append(V)
    sol = ctx.solve(Vs, 0.0, 12.0, mu, cap, FINE, level_capacity=64)
    for p, V in enumerate(Vs):
        n = int(sol.n_out[p])
        assert n == int(sol.n_total[p]) > 15
        E = sol.energy[p, :n]
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)) and np.all(sol.status[p, :n] == 0)
        last = V.min() + FINE * ((cap - V.min()) / FINE)
        c = W.count(V, h, mu, np.concatenate([E - 1e-10, E + 1e-10, [last]]))
        assert np.array_equal(c[:n], np.arange(n)) and np.array_equal(c[n:2 * n], np.arange(n) + 1)
        assert c[-1] == n
