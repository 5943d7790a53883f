"""Inputs changed in place between two calls, the arrays and their tables staying
where they are: the later call gives the result of the new values.

  * tj_get_hamiltonian: couplings, site energies and the places of a basis's
    states, against the oracle on the same inputs (<= 1e-12 of the largest entry);
  * tj_update_trun (a measurement operator's step): the operator doubled, so
    exactly twice the result;
  * tj_truncation: entries of the wavefunction changed, against the same values
    in another array (the same bits).
"""
import ctypes as C
import os

import numpy as np
import pytest

from grand_sql_tj_b200 import synth
from grand_sql_tj_b200.structs import Basis, BasisMap, TjBlockResult, Wave, WaveSector, call_block_result, call_model_result

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(product_lib):
    from grand_sql_tj_b200.lib import Context
    c = Context(0)
    yield c
    c.close()


def _data(m):
    d = [sb.mat.reshape(-1, order="F") for b in [m.ham] + [getattr(s, k) for s in m.sub for k in
                                                          ("elec_up", "elec_down", "spin_sd", "num_sn")] for sb in b.subs]
    return np.concatenate(d)


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("what", ["esite", "jt", "jd", "jn", "basis"])
def test_renorm(ctx, oracle_lib, product_lib, what, side):
    from oracle import oracle
    oracle.set_threads(os.cpu_count() or 1)
    rc = synth.renorm_case("cyl4", side=side)
    pp, pb, pt = rc.pre.pack(), rc.basis.pack(), rc.trun.pack()

    def call():
        r, m = call_model_result(lambda res: product_lib.tj_get_hamiltonian(
            ctx.h, C.byref(rc.lat.c), rc.side, rc.mshift, C.byref(pp.c), C.byref(pb.c), C.byref(pt.c), res))
        assert r == 0
        return _data(m)

    first = call()
    basis = rc.basis
    if what == "basis":
        # two equally large parts of each sector change places
        maps = []
        for i, m in enumerate(basis.maps):
            subs = list(m.subs)
            pair = [(a, b) for a in range(len(subs)) for b in range(a) if subs[a][1] == subs[b][1]][:1]
            for a, b in pair:
                subs[a], subs[b] = (subs[b][0],) + subs[a][1:], (subs[a][0],) + subs[b][1:]
                ca, cb = pb.maps[pb.sub[i].first + a], pb.maps[pb.sub[i].first + b]
                ca.spos, cb.spos = cb.spos, ca.spos
            maps.append(BasisMap(m.new_num_up, m.new_num_down, subs))
        basis = Basis(basis.len, maps)
    else:
        getattr(rc.lat, what)[:] *= 1.5
        if what == "jn":
            rc.lat.jn[:] += 0.25
    second = call()
    ref = _data(oracle.get_hamiltonian(rc.lat, rc.side, rc.mshift, rc.pre, basis, rc.trun))
    assert np.max(np.abs(ref - first)) > 1e-6 * np.max(np.abs(ref))   # the change matters
    assert np.max(np.abs(second - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_measurement_operator(ctx, product_lib):
    rc = synth.renorm_case("cyl4", side=0)
    ori, trun = rc.pre.ham, synth.random_trun(
        Basis(rc.pre.len, [BasisMap(s.num_up, s.num_down, [(0, s.mat.shape[0], 0, 0, 0, 0)]) for s in rc.pre.ham.subs]),
        30, np.random.default_rng(3))
    po, pt = ori.pack(), trun.pack()

    def call():
        r, b = call_block_result(lambda res: product_lib.tj_update_trun(ctx.h, 1, C.byref(po.c), C.byref(pt.c), res))
        assert r == 0
        return np.concatenate([s.mat.reshape(-1, order="F") for s in b.subs])

    first = call()
    po.data *= 2.0
    assert np.max(np.abs(first)) > 0 and np.array_equal(call(), 2.0 * first)
    # a first call that no second followed
    res = TjBlockResult()
    assert product_lib.tj_update_trun(ctx.h, 1, C.byref(po.c), C.byref(pt.c), C.byref(res)) == 0
    po.data *= 2.0
    assert np.array_equal(call(), 4.0 * first)


def test_truncation(ctx):
    rng = np.random.default_rng(7)
    n = 90
    w = Wave(3, 3, [WaveSector(4, 0, 4, 0, n, n)], rng.standard_normal(n * n))
    for at in range(4000, 4006):   # one entry at a time
        _, b = ctx.truncation(w, 0, 20, 20, 0.0)
        before = b.subs[0].mat.copy()
        w.data[at] += 0.5
        _, got = ctx.truncation(w, 0, 20, 20, 0.0)
        _, ref = ctx.truncation(w.copy(), 0, 20, 20, 0.0)
        assert np.array_equal(got.subs[0].mat, ref.subs[0].mat)
        assert not np.array_equal(got.subs[0].mat, before)
