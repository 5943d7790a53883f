"""The renormalisation cut into steps along its uploads: one step, two, and the
most there are, against the oracle (1e-12 of the largest entry, as the whole
pass is held to), with the operators from the host and from copies kept on the
device (the same bits: the steps are then bound by nothing but their order),
and into memory that is not page-locked."""
import os

import numpy as np
import pytest

from grand_sql_tj_b200 import synth
from test_gpu_renorm import _arrays, _same, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [60, 500, 640, 900, 1500])   # 0.2, 7, 12, 23 and 62 MB of operators
def test_steps(ctx, oracle_lib, monkeypatch, m):  # noqa: F811
    from grand_sql_tj_b200 import lib
    from oracle import oracle
    oracle.set_threads(os.cpu_count() or 1)
    sb = synth.make_superblock(24, 4, 47, 47, m, 84, 5)
    trun = synth.random_trun(sb.sys_bs, m, np.random.default_rng(m))
    args = (sb.lat, 0, 0, sb.sys, sb.sys_bs, trun)
    ref = oracle.get_hamiltonian(*args)
    got = ctx.get_hamiltonian(*args)
    _same(got, ref, 1e-12)
    first = _arrays(got)[1]
    lib.lib().tj_set_residency(ctx.h, 4.0)
    try:
        for _ in range(2):
            assert np.array_equal(_arrays(ctx.get_hamiltonian(*args))[1], first)
    finally:
        lib.lib().tj_set_residency(ctx.h, 0.0)
    monkeypatch.setattr(lib.HOST_POOL, "get", lambda n: np.empty(n))
    assert np.array_equal(_arrays(ctx.get_hamiltonian(*args))[1], first)
