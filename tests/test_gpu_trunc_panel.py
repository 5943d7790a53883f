"""The tridiagonal reductions: of a small sector in one CTA's shared memory at
the row counts of its lanes; the panelled one of a large sector: whole and
partial last panels, owned columns that are all, partly or from some panel on resident, and
the smallest trailing blocks a cluster shares; the tolerances are those of the
truncation's other stages (a backward error of 20 n eps ||rho||).
"""
import numpy as np
import pytest

from test_gpu_trunc_stages import _check, _psi, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kept", [(191, 191), (192, 192), (193, 40), (208, 60), (257, 100), (320, 320), (321, 50), (335, 335), (336, 20), (337, 60), (500, 100), (632, 30),
                                    (640, 30), (700, 700), (900, 25), (2200, 12)])
def test_panels(ctx, n, kept):  # noqa: F811
    _check(ctx, _psi(n, n, np.exp(-4.0 * np.arange(n) / n), n), kept)


# by one CTA: in shared memory, one or two rows a lane; above 64 states in L2
@pytest.mark.parametrize("n,kept", [(1, 1), (2, 2), (3, 3), (16, 9), (17, 17), (32, 32), (33, 20), (64, 64), (65, 30), (96, 96),
                                    (97, 50), (128, 128), (159, 70), (160, 160)])
def test_one_cta(ctx, n, kept):  # noqa: F811
    _check(ctx, _psi(n, n, np.exp(-4.0 * np.arange(n) / n), n), kept)


@pytest.mark.parametrize("n", [150, 330, 660])
def test_panels_deflate(ctx, n):  # noqa: F811
    """Reflectors that vanish: a matrix that is diagonal but for a block."""
    rng = np.random.default_rng(n)
    d = np.diag(rng.uniform(0.1, 1.0, n))
    d[60:100, 60:100] = rng.standard_normal((40, 40))
    d[n - 30:, n - 30:] = 0.0
    _check(ctx, d, n // 3)
