"""The set-up kernels at the edges of their tiles (2048 points) and blocks (32):
wells whose cut-offs, minimum or inner barrier lie on, just before and just
after them, and a minimum on the grid's end points.  The plain method against
the FP64 oracle, whose energies it must give to the last bit: they depend on
the cut-offs, the twist index, the trial ladder and the turning points found
through the block minima; the fast method against the plain one (level totals
equal, energies within the project's bar of 1e-10 Hartree)."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _well(N, c, lo, hi, barrier=None):
    """unit spacing and mass: V up to 3 above the minimum is inside the cut-off"""
    i = np.arange(N, dtype=np.float64)
    V = 0.5 * 0.0025 * (i - c) ** 2 - 0.3
    V[:lo] = 50.0
    V[hi + 1:] = 50.0
    if barrier is not None:
        V[barrier] = 40.0
    return V


@pytest.mark.parametrize("N", [33, 64, 65, 2047, 2048, 2049, 4095, 4096, 4097, 6200])
def test_tile_and_block_edges(ctx, N):
    wells = [_well(N, 0.5 * (N - 1), 0, N - 1), _well(N, 0, 0, N - 1), _well(N, N - 1, 0, N - 1),
             _well(N, N // 2, N // 2 - 9, N // 2 + 8)]
    for e in (32, 2048, 4096):
        for c in (e - 1, e, e + 1):
            for lo, hi in ((0, N - 1), (e - 12, e + 11), (e - 1, N - 1), (e, N - 1), (e + 1, N - 1), (0, e - 1), (0, e)):
                lo = max(lo, 0)
                if hi < N and lo < c < hi:
                    wells.append(_well(N, c, lo, hi))
    n_smooth = len(wells)  # (the wells below have a one-point barrier)
    for e in (32, 2048, 4096):
        for k in (e - 1, e):
            if 4 <= k < N - 4:
                wells.append(_well(N, k + 3, 0, N - 1, barrier=k))
    r1 = float(N - 1)
    args = (wells, 0.0, r1, 1.0, 0.14, 64)
    refs = O.solve_batch(*args)
    sol = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=64)
    fast = ctx.solve(*args, method=capi.METHOD_FAST_FP32C, level_capacity=64)
    assert sum(x.n_total for x in refs) > 0
    for p, ref in enumerate(refs):
        n = int(sol.n_out[p])
        assert int(sol.n_total[p]) == ref.n_total, p
        assert np.array_equal(sol.energy[p, :n], ref.energy), p
        if p >= n_smooth:
            continue  # (a one-point barrier: the set-up's flag is what it is for)
        assert int(fast.n_total[p]) == ref.n_total, p
        if n:
            assert np.max(np.abs(fast.energy[p, :n] - ref.energy)) < 1e-10, p
