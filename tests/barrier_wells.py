"""Wells with a barrier inside the grid, up to where f = 1 + T (T = a (E - V)) is
negative, and their levels from CPU restatements of the discrete problem.

With u = f psi the problem is J u = 0, J = tridiag(-1, g / f, -1), g = 2 - 10 T.
J = 12 (F^-1 - B), F = diag(f), B = tridiag(1, 10, 1) / 12, and by the two Schur
complements of [[F^-1, I], [I, B^-1]] the number of negative pivots of J is the
number of levels below E plus the number of negative f."""
from __future__ import annotations

import numpy as np

CAP = 0.14  # energy cap of the wells below; a = 1/6 (unit mass and spacing)
F_BARRIER = (0.1, -0.1, -1.0, -5.7, -1e3)
WIDTHS = (1, 2, 3, 20)


def wells():
    """Harmonic wells of ~14 levels cut in two unequal parts by a barrier of some
    points where f takes the value at half the cap; (V, barrier slice, f) each."""
    out = []
    N = 161
    i = np.arange(N, dtype=np.float64)
    for at in (68, 90):
        for n in WIDTHS:
            for f in F_BARRIER:
                V = 0.5 * 1e-4 * (i - 79.3) ** 2
                V[at:at + n] = 0.5 * CAP + 6.0 * (1.0 - f)
                out.append((V, slice(at, at + n), f))
    return out


def cuts(V, h, mu):
    """The Dirichlet cut-offs and a."""
    a = mu * h * h / 6.0
    inside = np.nonzero(a * (V - V.min()) <= 0.5)[0]
    return max(1, int(inside[0])), min(V.size - 2, int(inside[-1])), a


def count(V, h, mu, E):
    """Levels below each energy of E: negative pivots of J less negative f."""
    i0, i1, a = cuts(V, h, mu)
    E = np.atleast_1d(np.asarray(E, np.float64))
    n = np.zeros(E.size, np.int64)
    d = np.full(E.size, np.inf)
    for i in range(i0, i1 + 1):
        T = a * (E - V[i])
        f = 1.0 + T
        d = (2.0 - 10.0 * T) / f - 1.0 / d
        n += (d < 0.0).astype(np.int64) - (f < 0.0)
    return n


def dense(V, h, mu, cap):
    """Levels below cap and their wavefunctions (sum psi^2 h = 1, positive next to
    the inner wall), by diagonalisation of diag(V) - B^-1 D2 / (2 mu h^2)."""
    i0, i1, _ = cuts(V, h, mu)
    n = i1 - i0 + 1
    one = np.ones(n - 1)
    B = (np.diag(np.full(n, 10.0)) + np.diag(one, 1) + np.diag(one, -1)) / 12.0
    D2 = np.diag(np.full(n, -2.0)) + np.diag(one, 1) + np.diag(one, -1)
    H = np.diag(V[i0:i1 + 1]) - np.linalg.solve(B, D2) / (2.0 * mu * h * h)
    E, X = np.linalg.eigh(0.5 * (H + H.T))
    k = int(np.searchsorted(E, cap))
    psi = np.zeros((k, V.size))
    psi[:, i0:i1 + 1] = X[:, :k].T / np.sqrt(h)
    for row in psi:
        row *= np.sign(row[np.argmax(np.abs(row) > 1e-6 * np.abs(row).max())])
    return E[:k], psi
