"""The plain FP64 method on wells with a barrier inside the grid, up to where
f = 1 + T is negative, and the Lennard-Jones parameter gradient at negative r:
both take the reciprocal of a negative number.

Energies, node counts and status are the oracle's (to the bit); the wavefunctions
are compared at the levels where the oracle's energy is the dense solution's to
1e-10 (its counts are off where a solution has a node beside such a barrier).
Tolerance: both are stitched at an energy within the bracket of 1e-12, so they
differ by at most ~1e-12 over the gap to the next level, 2.7e-4 at least: the
project's bar of 1e-8 in L2 holds it."""
from __future__ import annotations

import numpy as np
import pytest

import barrier_wells as W
from epseon_backend_gb300 import capi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_wavefunctions_across_a_barrier(ctx):
    wells = W.wells()
    args = ([w[0] for w in wells], 0.0, 160.0, 1.0, W.CAP, 512)
    refs = O.solve_batch(*args, want_psi=True)
    sol = ctx.solve(*args, method=capi.METHOD_PLAIN_FP64, level_capacity=32, want_psi=True)
    negative = 0
    for p, ((V, _, f), ref) in enumerate(zip(wells, refs)):
        n = int(sol.n_out[p])
        assert int(sol.n_total[p]) == ref.n_total and n == ref.n_total, p
        assert np.array_equal(sol.energy[p, :n], ref.energy), p
        E, psi = W.dense(V, 1.0, 1.0, W.CAP)
        assert E.size == n, p
        good = np.nonzero(np.abs(ref.energy - E) < 1e-10)[0]
        assert good.size >= 1, p
        negative += good.size if f < 0.0 else 0
        got = sol.wavefunctions(p)
        assert np.array_equal(sol.nodes[p, good], good), p
        assert np.all(sol.status[p, good] == 0), p
        for v in good:
            assert np.linalg.norm(got[v] - ref.psi[v]) < 1e-8, (p, v)
            assert min(np.linalg.norm(got[v] - psi[v]), np.linalg.norm(got[v] + psi[v])) < 1e-8, (p, v)
    assert negative > 100


@pytest.mark.parametrize("r0, r1", [(-12.0, -2.6), (2.6, 12.0)])
def test_lennard_jones_gradient_at_negative_r(ctx, r0, r1):
    """against the closed-form derivatives in FP64: sums of the terms' rounding"""
    N, eps, sigma = 4099, 0.05, 3.0
    row = np.concatenate([[eps, sigma], np.zeros(10)])
    g = np.random.default_rng(5).standard_normal(N) / N
    gP = ctx.tabulate_adjoint(np.array([synth.KIND_LJ]), row[None], np.array([N], np.int32), np.array([r0]),
                              np.array([r1]), g)[0]
    s6 = (sigma / np.linspace(r0, r1, N)) ** 6
    terms = np.array([4.0 * (s6 * s6 - s6) + 1.0, 4.0 * eps * (12.0 * s6 * s6 - 6.0 * s6) / sigma]) * g
    assert np.all(np.abs(gP[:2] - terms.sum(1)) <= 1e-13 * np.abs(terms).sum(1))
    assert np.all(gP[2:] == 0.0)
