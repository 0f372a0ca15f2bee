"""Tabulation and its adjoint at the sizes where their index arithmetic can go
wrong: few knots and many, grids shorter and longer than the knots, tile and
block remainders, the spline's exact knots.  Values against the host FP64
tabulation (1e-11 relative, the project's bar), gradients against central
differences of it (1e-7 relative)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

SPLINE = np.array([0.1, 1.0, 2.0, 0.01, 0.3, 2.5, -0.008, 0.2, 3.0, 0.0, 0.0, 0.0])
MORSE = np.concatenate([[0.08, 1.2, 1.8], np.zeros(9)])
LJ = np.concatenate([[0.05, 3.0], np.zeros(10)])
N = np.array([2, 3, 5, 63, 64, 65, 255, 257, 1023, 1024, 1025, 2047, 2049, 4099, 70001], np.int32)


@pytest.mark.parametrize("n_knots", [4, 5, 29, 64, 1023, 1024, 2500])
def test_values_at_awkward_sizes(ctx, n_knots):
    kinds, P, sizes = [], [], []
    for kind, row in ((synth.KIND_SPLINE, SPLINE), (synth.KIND_MORSE, MORSE), (synth.KIND_LJ, LJ)):
        kinds += [kind] * N.size
        P += [row] * N.size
        sizes += list(N)
    sizes = np.array(sizes, np.int32)
    r0, r1 = np.full(sizes.size, 0.5), np.full(sizes.size, 20.0)
    V = ctx.tabulate(np.array(kinds), np.array(P), sizes, r0, r1, n_knots=n_knots)
    for i in range(sizes.size):
        Vh = synth.tabulate_params(kinds[i], P[i], sizes[i], 0.5, 20.0, n_knots)
        assert np.max(np.abs(V[i] - Vh) / np.maximum(1.0, np.abs(Vh))) < 1e-11, (kinds[i], sizes[i])


@pytest.mark.parametrize("n_knots", [4, 29, 1024, 2500])
def test_adjoint_at_awkward_sizes(ctx, n_knots):
    rng = np.random.default_rng(n_knots)
    for kind, row, used in ((synth.KIND_SPLINE, SPLINE, 9), (synth.KIND_MORSE, MORSE, 3), (synth.KIND_LJ, LJ, 2)):
        sizes = N[2:]
        n = sizes.size
        # r_min inside the well: V and its derivatives of one magnitude
        r0, r1 = np.full(n, 1.5 if kind != synth.KIND_LJ else 2.6), np.full(n, 12.0)
        g = [rng.standard_normal(s) / s for s in sizes]
        gP = ctx.tabulate_adjoint(np.full(n, kind), np.tile(row, (n, 1)), sizes, r0, r1, np.concatenate(g), n_knots)
        again = ctx.tabulate_adjoint(np.full(n, kind), np.tile(row, (n, 1)), sizes, r0, r1, np.concatenate(g), n_knots)
        assert np.array_equal(gP, again)
        assert np.all(gP[:, used:] == 0.0)
        for i in range(n):
            d = np.zeros(12)
            d[:used] = rng.uniform(0.5, 1.5, used) * np.maximum(np.abs(row[:used]), 1e-2)

            def f(t):
                return float(g[i] @ synth.tabulate_params(kind, row + t * d, sizes[i], r0[i], r1[i], n_knots))

            fd = (f(1e-5) - f(-1e-5)) / 2e-5
            assert abs(gP[i] @ d - fd) <= 1e-7 * max(abs(fd), np.abs(gP[i] * d).max()), (kind, sizes[i])
