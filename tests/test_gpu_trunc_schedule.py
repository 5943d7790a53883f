"""Which sectors a cluster reduces and which one CTA, when not all clusters run at
a time: a call's tridiagonal stage takes no jump where its sectors pass the size
from which a cluster reduces one faster (191 and 200 states, 21 sectors: the
work grows by 15 %, half as much time again is allowed), and sectors of sizes
between, reduced by either, give their eigenvectors.

Tolerances of the second as in the truncation's stages: residuals and the
distance of the kept weight from the sum of the largest eigenvalues within
20 n eps ||rho||, orthonormal to 1e-12.
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


def _wave(dims, k, seed):
    rng = np.random.default_rng(seed)
    parts = [rng.standard_normal((n, k)) * np.exp(-3.0 * np.arange(k) / k) for n in dims]
    x = np.concatenate([a.T.reshape(-1) for a in parts])
    x /= np.linalg.norm(x)
    return Wave(3, 3, [WaveSector(4 + i, 0, 4, 0, n, k) for i, n in enumerate(dims)], x)


def test_no_jump_at_the_cluster_size(ctx):
    def stage(n):
        t = []
        for r in range(5):
            ctx.truncation(_wave([n] * 21, 30, r), 0, 40, 40, 0.0)
            t.append(ctx.stats().trunc_ms_tridiag)
        return min(t)

    assert stage(200) <= 1.5 * stage(191)


# all by one CTA; the largest by clusters; enough clusters for all
@pytest.mark.parametrize("dims", [[200] * 21, [319, 256, 193, 192] * 8, [340, 320] + [319, 250, 192, 130, 64, 33] * 7,
                                  [400, 300, 200, 100]])
def test_sizes_between(ctx, dims):
    k, kept = 400, 40 * len(dims)
    w = _wave(dims, k, 11)
    r, b = ctx.truncation(w, 0, kept, kept, 0.0)
    assert r.num_state in (kept, kept + 1)
    rho = [w.sector(i) @ w.sector(i).T for i in range(len(dims))]
    ev = [np.linalg.eigvalsh(x) for x in rho]
    got = {s.num_up: s.mat for s in b.subs}
    assert sum(u.shape[1] for u in got.values()) == r.num_state
    top = np.sort(np.concatenate(ev))[-r.num_state:]
    weight = tols = 0.0
    for i, n in enumerate(dims):
        u = got.get(4 + i)
        if u is None:
            continue
        tol = 20 * n * 2.0 ** -52 * ev[i][-1]
        assert np.max(np.abs(u.T @ u - np.eye(u.shape[1]))) <= 1e-12
        ru = rho[i] @ u
        lam = np.sum(u * ru, axis=0)
        assert np.max(np.linalg.norm(ru - u * lam, axis=0)) <= tol
        weight += lam.sum()
        tols += tol * u.shape[1]
    assert abs(weight - top.sum()) <= tols
