"""The stages of the truncation at the sizes and spectra where they change
path: the back-transformation's block counts and row tiles (a sector of 1 to
1536 states, and above), the tridiagonal reduction by one CTA and by a
cluster, the orthonormalisation by products (separated eigenvalues) and
vector by vector (clusters, null spaces, a reducible matrix).

The wavefunction has one sector of n states with given singular values.
Tolerances: the kept vectors u are those of a matrix within p(n) eps ||rho|| of
rho, p(n) = 20 n for a Householder reduction in FP64, so the residual
||rho u - (u.rho u) u|| is below that, and so is the distance of the kept
weight from the sum of the largest eigenvalues; orthonormal to 1e-12 (as the
parity tests of the truncation ask).
"""
import numpy as np
import pytest

from grand_sql_tj_b200.structs import Wave, WaveSector

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(product_lib):
    from grand_sql_tj_b200.lib import Context
    c = Context(0)
    yield c
    c.close()


def _check(ctx, psi, kept):
    n, m = psi.shape
    psi = psi / np.linalg.norm(psi)
    w = Wave(3, 3, [WaveSector(4, 0, 4, 0, n, m)], np.ascontiguousarray(psi.T).reshape(-1))
    rho = psi @ psi.T
    r, b = ctx.truncation(w, 0, kept, kept, 0.0)
    # the keep rule takes states from kept_min on while weight is left, at least one
    # (den_mat.f90:263-282; a discarded weight of rounding size may have either sign)
    assert r.num_state in ((kept,) if kept >= n else (kept, kept + 1))
    kept = r.num_state
    u = b.subs[0].mat
    assert u.shape == (n, kept)
    assert np.max(np.abs(u.T @ u - np.eye(kept))) <= 1e-12
    ev = np.linalg.eigvalsh(rho)
    tol = 20 * n * 2.0 ** -52 * ev[-1]
    ru = rho @ u
    lam = np.sum(u * ru, axis=0)
    assert np.max(np.linalg.norm(ru - u * lam, axis=0)) <= tol
    assert abs(np.sum(lam) - np.sum(ev[n - kept:])) <= kept * tol
    top = np.argmax(np.abs(u), axis=0)
    assert np.all(u[top, np.arange(kept)] > 0)


def _psi(n, m, sv, seed):
    rng = np.random.default_rng(seed)
    k = len(sv)
    q = np.linalg.qr(rng.standard_normal((n, k)))[0]
    p = np.linalg.qr(rng.standard_normal((m, k)))[0]
    return (q * sv) @ p.T


@pytest.mark.parametrize("n,kept", [(1, 1), (2, 2), (3, 1), (8, 5), (16, 16), (17, 9), (33, 20), (129, 60), (257, 130),
                                    (319, 100), (320, 100), (513, 64), (770, 300), (1025, 40), (1290, 33), (1537, 24)])
def test_separated(ctx, n, kept):
    _check(ctx, _psi(n, n, np.exp(-5.0 * np.arange(n) / n), n), kept)


@pytest.mark.parametrize("n", [5, 40, 200, 350])
def test_clusters_and_null_space(ctx, n):
    m = max(1, n // 2)
    # rank n / 2, more kept than that
    _check(ctx, _psi(n, m, np.exp(-3.0 * np.arange(m) / m), n), m + n // 5)
    # all weights equal
    _check(ctx, _psi(n, n, np.ones(n), n + 1), n)
    # weights falling far below the accuracy
    _check(ctx, _psi(n, n, np.exp(-40.0 * np.arange(n) / n), n + 2), n // 2)


def test_reducible(ctx):
    rng = np.random.default_rng(2)
    d = np.zeros((60, 60))
    d[np.arange(60), np.arange(60)] = rng.uniform(0.1, 1.0, 60)   # diagonal: no reflector at all
    _check(ctx, d, 30)
    d[20:40, 20:40] = rng.standard_normal((20, 20))
    d[40:, 40:] = 0.0
    _check(ctx, d, 45)
