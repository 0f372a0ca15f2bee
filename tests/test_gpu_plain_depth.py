"""The plain method's bisection at every depth of its tree (how many halvings a
march takes follows from the number of levels): copies of three small Morse
wells, from a few levels to more than the depths' limits, against the FP64
oracle.  Same operations as the oracle's: energies equal to the bit, node
counts and wavefunctions as the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 12, 50, 100, 300, 700])
def test_bisection_depths_are_bit_exact(ctx, copies):
    r = np.linspace(0.5, 14.0, 601)
    wells = [synth.morse(r, De, 1.0, 2.0) for De in (0.05, 0.08, 0.1)]
    mu, cap = 1500.0, 0.045
    refs = O.solve_batch(wells, 0.5, 14.0, mu, cap, 256, want_psi=True)
    V = wells * copies
    sol = ctx.solve(V, 0.5, 14.0, mu, cap, 256, method=capi.METHOD_PLAIN_FP64, level_capacity=24, want_psi=True)
    total = int(sol.n_out.sum())
    assert total == copies * sum(x.n_total for x in refs)
    h = r[1] - r[0]
    for p in range(len(V)):
        ref = refs[p % 3]
        n = int(sol.n_out[p])
        assert np.array_equal(sol.energy[p, :n], ref.energy), p
        assert np.array_equal(sol.nodes[p, :n], np.arange(n)), p
        if p < 3 or p >= len(V) - 3:
            err = np.sqrt(np.sum((sol.wavefunctions(p) - ref.psi) ** 2, axis=1) * h)
            assert err.max() < 1e-8
