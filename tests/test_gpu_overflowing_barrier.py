"""The plain method's level totals where the recurrence overflows between two
renormalisations (barriers of 1 to 40 points up to 1e300): its states become
infinities and NaN there, and as in the oracle a NaN is not negative in the
counts.  Equal to the oracle's at every energy cap."""
from __future__ import annotations

import numpy as np
import pytest

from epseon_backend_gb300 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [0.02, 0.05, 0.09, 0.14])
def test_totals_through_infinities(ctx, cap):
    i = np.arange(161, dtype=np.float64)
    Vs = []
    for top in (1e3, 1e12, 1e20, 1e40, 1e160, 1e300):
        for n in (1, 2, 40):
            for at in (50, 90):
                V = 0.5 * 1e-4 * (i - 79.3) ** 2
                V[at:at + n] = top
                Vs.append(V)
    args = (Vs, 0.0, 160.0, 1.0, cap, 256)
    refs = O.solve_batch(*args)
    sol = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=256)
    assert [int(x) for x in sol.n_total] == [r.n_total for r in refs]
