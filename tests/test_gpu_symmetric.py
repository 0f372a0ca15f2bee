"""Node counts of symmetric wells on grids with a point at the centre, where
every odd level's wavefunction is zero to rounding: on a strip or chunk boundary
of the group passes the two threads that meet there must not both count the sign
change, nor neither of them.  Levels 0 .. n - 1 exactly, no status flag, and the
energies within the project's bar of 1e-10 Hartree of the plain method's."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi

pytestmark = pytest.mark.gpu

WARP, CTA = 1 << 24, 1


@pytest.mark.parametrize("wait_polls", [0, 1 << 22])
@pytest.mark.parametrize("long_window", [0, WARP, CTA])
def test_symmetric_wells(ctx, long_window, wait_polls):
    V, mu = [], []
    for N in (129, 257, 385, 513, 545, 769, 1025, 1537, 2049, 3073, 4097):
        r = np.linspace(-1.0, 1.0, N)
        for s, c4 in ((1.0, 0.0), (1.3, 0.0), (0.7, 2.0), (1.0, 1.0)):
            V.append(s * 0.5 * r * r + c4 * r ** 4)
            mu.append(2.0 * (N - 1))
    args = (V, -1.0, 1.0, np.array(mu), 0.45, 200)
    ref = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=100)
    sol = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=100, want_psi=True, long_window=long_window,
                    wait_polls=wait_polls)
    assert np.array_equal(sol.n_total, ref.n_total)
    assert int(ref.n_out.sum()) > 200
    for p in range(len(V)):
        n = int(ref.n_out[p])
        assert n > 0
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), (p, sol.nodes[p, :n])
        assert np.all(sol.status[p, :n] == 0), p
        assert np.max(np.abs(sol.energy[p, :n] - ref.energy[p, :n])) < 1e-10, p


def test_symmetric_wells_on_clusters(ctx):
    V, mu = [], []
    for N in (32769, 40961, 65537):
        r = np.linspace(-1.0, 1.0, N)
        V.append(0.5 * r * r)
        mu.append(2000.0)
    sol = ctx.solve(V, -1.0, 1.0, np.array(mu), 0.3, 400, level_capacity=60, want_psi=True)
    for p in range(3):
        n = int(sol.n_out[p])
        assert n >= 10
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), p
        assert np.all(sol.status[p, :n] == 0), p
