"""The Lanczos solve that stops because nothing is left of the next vector
(|beta| <= lanzero, code/tjsq/eigen.f90:2-175): the start vector spans an
invariant space, beta is exactly zero, and the vector computed from it, which
the result does not use, is 0 / 0.  In FP64 and in split precision, for a vector
short enough for one cluster and for a longer one: one iteration, the Rayleigh
quotient and the normalised start vector.  A start vector that does hold a NaN
is refused in both.
"""
import numpy as np
import pytest

from grand_sql_tj_b200 import synth
from grand_sql_tj_b200.structs import Wave

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["fp64", "split"])
def ctx(product_lib, request):
    from grand_sql_tj_b200.lib import TJ_PREC_OZAKI, Context
    c = Context(0)
    if request.param == "split":
        c.set_precision(TJ_PREC_OZAKI, 5)
    yield c
    c.close()


def test_one_entry(ctx):
    sb = synth.make_superblock(16, 2, 15, 15, 6, 28, 17)
    one = [s for s in sb.wave.sectors if s.sys_dim * s.env_dim == 1][:1]
    w = Wave(sb.wave.sys_len, sb.wave.env_len, one, np.array([-3.0]))
    h = ctx.model_wave(sb, w).data[0] / -3.0
    e, it, x = ctx.lanczos_memo_new(sb, 2e-5, start=w)
    assert it == 1 and abs(x.data[0]) == 1.0
    # the same arithmetic but for the vector's scale, 3 and 1: rounding of FP64 or of 5 slices
    assert abs(e - h) <= 1e-9 * max(1.0, abs(h))


# 1434 entries by one cluster, 49,347 by the grid's kernels
@pytest.mark.parametrize("m", [64, 377])
def test_zero_operator(ctx, m):
    sb = synth.make_superblock(16, 2, 15, 15, m, 28, 17)
    for model in (sb.sys, sb.env):
        for b in [model.ham] + [getattr(s, k) for s in model.sub for k in ("elec_up", "elec_down", "spin_sd", "num_sn")]:
            for s in b.subs:
                s.mat[:] = 0.0
    for a in (sb.lat.jt, sb.lat.jz, sb.lat.jd, sb.lat.jn, sb.lat.esite):
        a[:] = 0.0
    e, it, x = ctx.lanczos_memo_new(sb, 2e-5)
    assert it == 1 and e == 0.0
    start = sb.wave.data / np.linalg.norm(sb.wave.data)
    assert np.max(np.abs(np.abs(x.data) - np.abs(start))) <= 1e-14


@pytest.mark.parametrize("m", [64, 377])
def test_nan_start(ctx, m):
    from grand_sql_tj_b200.lib import TjError
    sb = synth.make_superblock(16, 2, 15, 15, m, 28, 17)
    bad = sb.wave.copy()
    bad.data[bad.dim // 2] = np.nan
    with pytest.raises(TjError) as e:
        ctx.lanczos_memo_new(sb, 2e-5, start=bad)
    assert e.value.code == 7
    good, _, _ = ctx.lanczos_memo_new(sb, 2e-5)
    assert np.isfinite(good)
