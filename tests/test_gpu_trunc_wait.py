"""The waits of the cluster's tridiagonal reduction run out: with the limit at 0 s
(tj_set_wait_limit) the first wait for data that has not come yet gives up, the
CTAs run through their steps without exchanging anything more, the call returns
TJ_ERR_TIMEOUT, and the same context and a fresh one truncate correctly after it
(the check and its tolerances are those of the truncation's stages).  Sectors
that one CTA reduces alone do not wait.
"""
import numpy as np
import pytest

from test_gpu_trunc_stages import _check, _psi

pytestmark = pytest.mark.gpu


# one panel boundary after another, the last rows and the resident columns: 321, 900 states
@pytest.mark.parametrize("n", [321, 900])
def test_wait_limit_runs_out(product_lib, n):
    from grand_sql_tj_b200.lib import Context, TjError
    psi = _psi(n, n, np.exp(-4.0 * np.arange(n) / n), n)
    c = Context(0)
    try:
        for _ in range(2):
            c.set_wait_limit(0.0)
            with pytest.raises(TjError) as e:
                _check(c, psi, 40)
            assert e.value.code == 6
            _check(c, psi[:100], 20)
            c.set_wait_limit(2.0)
            _check(c, psi, 40)
    finally:
        c.close()
    fresh = Context(0)
    try:
        _check(fresh, psi, 40)
    finally:
        fresh.close()
