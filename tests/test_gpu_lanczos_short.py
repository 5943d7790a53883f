"""The Lanczos iteration on both sides of the length up to which one
thread-block cluster takes its vector steps, and at its smallest: fewer entries
than the cluster has CTAs, one and two entries a CTA.

The oracle is the same recurrence in numpy over the H*psi entry point.  With
one start vector and threshold both stop at the same step, or one apart where a
step's change of the Ritz value is the threshold to rounding: the energies agree
to the threshold plus 1e-12 |E|, the vectors to an overlap of 1 - 1e-8.
"""
import numpy as np
import pytest

from grand_sql_tj_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(product_lib):
    from grand_sql_tj_b200.lib import Context
    c = Context(0)
    yield c
    c.close()


def _lanczos(apply, start, lanzero):
    v = [start / np.linalg.norm(start)]
    w = apply(v[0])
    alpha, beta = [v[0] @ w], []
    ritz = alpha[0]
    while len(v) < 110:
        w = w - alpha[-1] * v[-1] - (beta[-1] * v[-2] if beta else 0.0)
        b = np.linalg.norm(w)
        if b <= lanzero:
            break
        w = w / b
        w = w - sum((x @ w) * x for x in v)
        v.append(w / np.linalg.norm(w))
        beta.append(b)
        w = apply(v[-1])
        alpha.append(v[-1] @ w)
        last, ritz = ritz, np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))[0]
        if abs(ritz - last) <= lanzero:
            break
    e, z = np.linalg.eigh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))
    return e[0], len(v), np.array(v).T @ z[:, 0]


# entries: 7, 32, 44, 1434, 49030 | 49347 (the cluster takes up to 49152)
@pytest.mark.parametrize("m", [6, 8, 12, 64, 376, 377])
@pytest.mark.parametrize("lanzero", [2e-5, 1e-10])
def test_lanczos_lengths(ctx, m, lanzero):
    sb = synth.make_superblock(16, 2, 15, 15, m, 28, 17)
    e_ref, it_ref, x_ref = _lanczos(lambda x: ctx.model_wave(sb, sb.wave.like(x)).data, sb.wave.data, lanzero)
    e, it, w = ctx.lanczos_memo_new(sb, lanzero)
    assert abs(it - it_ref) <= 1, (it, it_ref)
    assert abs(e - e_ref) <= lanzero + 1e-12 * abs(e_ref)
    assert abs(np.dot(w.data, x_ref)) / np.linalg.norm(x_ref) >= 1 - 1e-8
    assert abs(np.linalg.norm(w.data) - 1.0) < 1e-12
