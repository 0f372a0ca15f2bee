"""A replayed solve with other grid lengths in the same buffers (equal number of
potentials and points): the set-up's tile count, the longest grid, and with it
the scan's groups and the cluster list, belong to the captured graph.  The
context is warmed by a larger batch, so that no buffer grows in between and
drops the graph.  Results equal to the bit those of a context of its own."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth

pytestmark = pytest.mark.gpu

CAP = 96


def _solve(db, N, offsets, r0, r1):
    import torch

    db.N[:], db.offsets[:] = N, offsets
    for p in range(len(N)):
        V = synth.morse(np.linspace(r0, r1, N[p]), 0.1, 1.0 + 0.1 * p, 2.0)
        db.V[offsets[p]:offsets[p] + N[p]] = torch.from_numpy(V).cuda()
    for t in (db.energy, db.nodes, db.status, db.n_total):
        t.fill_(-7)
    db.solve()
    torch.cuda.synchronize()
    return [t.cpu().numpy().copy() for t in (db.n_total, db.energy, db.nodes, db.status)]


def _batch(ctx, total, n, N_max):
    h = (12.0 - 0.5) / (N_max - 1)
    mu = min(4000.0, 0.8 / (2 * 0.1 * h * h))
    layout = capi.Concatenated(np.zeros(total), np.zeros(n, np.int64), np.full(n, total // n, np.int32))
    return capi.DeviceBatch(ctx, layout, 0.5, 12.0, mu, 0.099, 600, CAP, want_psi=False)


@pytest.mark.parametrize("first, second", [
    (((4096, 4096), (0, 4096)), ((4097, 4095), (0, 4097))),        # a tile more
    (((4097, 4095), (0, 4097)), ((4096, 4096), (0, 4096))),        # a tile less
    (((4000, 9000), (0, 10000)), ((9000, 9000), (0, 10000))),      # fixed slots, another fill
    (((16000, 16000), (0, 16000)), ((20000, 12000), (0, 20000))),  # long enough for clusters
    (((66000, 65000), (0, 66000)), ((65500, 65500), (0, 65500))),  # no longer a CTA per trial energy
])
def test_replay_with_other_grid_lengths(first, second):
    total = max(o + N for part in (first, second) for N, o in zip(*part))
    warm, own = capi.Context(0), capi.Context(0)
    try:
        big = _batch(warm, 4 * total, 2, 2 * total)
        _solve(big, (2 * total, 2 * total), (0, 2 * total), 0.5, 12.0)
        a, b = _batch(warm, total, 2, 4000), _batch(own, total, 2, 4000)
        _solve(a, *first, 0.5, 12.0)
        got = _solve(a, *second, 0.5, 12.0)
        ref = _solve(b, *second, 0.5, 12.0)
        assert int(ref[0].min()) > 3
        for x, y in zip(got, ref):
            assert np.array_equal(x, y, equal_nan=True)
    finally:
        warm.close()
        own.close()
