"""Performance cases: the calls a DMRG program makes, step after step.

A sweep of the SU(2) t-J DMRG does, at every position of the chain, a Lanczos
solve (H*psi some tens of times on one compiled plan), the truncation of the
density matrix, the renormalisation of the block's operators into the new
basis and the prediction of the next start vector.  Each case is one such
call through the public interface (the Python Context, or the C ABI with the
tables and arrays such a program holds), with host arrays in and out as the
drop-in boundary has them.  The operators, truncation operators and
wavefunctions of a running sweep are arrays that the library itself wrote:
page-locked buffers of its host pool, all blocks of a model in one array;
`prepare` lays the inputs out the same way.

Sizes are those of the repository's configurations (2x6 and 2x16 ladders,
4x24 and 6x24 cylinders, m from tens to thousands, canonical and
grand-canonical labels).  `exact` evaluates the same quantities in plain
64-bit torch from the recoupling formulas of reduced SU(2) operators.
"""
import ctypes as C
import math
from functools import lru_cache

import numpy as np
import torch

from grand_sql_tj_b200 import lib, structs, synth
from grand_sql_tj_b200.lattice import Geometry


# ------------------------------------------------------------------ the cases
def _case(name, kind, nx, ny, m, holes, prec="fp64", slices=0, up_bias=1, t2=0.0, shift=0, side=0, lanzero=0.0,
          sigma=2.2):
    c = dict(kind=kind, nx=nx, ny=ny, m=m, holes=holes, prec=prec, slices=slices, up_bias=up_bias, t2=t2,
             shift=shift, side=side, lanzero=lanzero, sigma=sigma)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one H*psi of a program with its own eigensolver, the plan of the step kept: the smallest superblock
        # (2x6 ladder), where the call's fixed cost is everything
        _case("hpsi_ladder6_m24", "hpsi", 6, 2, 24, 2),
        # the same in the shipped reference mode (grand-canonical labels: few, larger sectors)
        _case("hpsi_gc4x6_m300", "hpsi", 6, 4, 300, 0, up_bias=0),
        # the benchmark's superblock in plain FP64
        _case("hpsi_cyl4x24_m2000", "hpsi", 24, 4, 2000, 12),
        # and in split precision (five slices)
        _case("hpsi_cyl4x24_m2000_s5", "hpsi", 24, 4, 2000, 12, "split", 5),
        # the six-leg cylinder with t', the largest superblock that prepares in seconds
        _case("hpsi_cyl6x24_m3000_s5", "hpsi", 24, 6, 3000, 18, "split", 5, t2=-0.2),
        # a whole Lanczos solve of a new step (plan, upload, iterations, Ritz vector): the CPU-size ladder in FP64
        _case("lanczos_ladder16_m256", "lanczos", 16, 2, 256, 4, lanzero=2e-5),
        # and the benchmark's end-to-end call in split precision
        _case("lanczos_cyl4x24_m2000_s5", "lanczos", 24, 4, 2000, 12, "split", 5, lanzero=2e-5),
        # truncation after the solve: a ladder step, and a cylinder step (the environment of a right-to-left sweep)
        # with the narrower spread of particle numbers, and so the larger sectors, that a converged run shows
        _case("trunc_ladder16_m256", "trunc", 16, 2, 256, 4),
        _case("trunc_cyl4x24_m2000", "trunc", 24, 4, 2000, 12, side=1, sigma=1.0),
        # renormalisation of the block's operators: off the middle of the chain, and the benchmark's size
        _case("renorm_cyl4x24_m500", "renorm", 24, 4, 500, 12, shift=3),
        _case("renorm_cyl4x24_m2000", "renorm", 24, 4, 2000, 12, side=1),
        # prediction of the next start vector
        _case("predict_cyl4x24_m2000", "predict", 24, 4, 2000, 12),
    ]


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "lanczos", "trunc", "renorm", "predict"])
    ny = rng.choice([2, 4, 4, 6])
    nx = {2: rng.randint(6, 24), 4: rng.randint(6, 24), 6: rng.randint(6, 24)}[ny]
    up_bias = 0 if rng.random() < 0.15 else 1
    hi = {"hpsi": 2200, "lanczos": 1400, "trunc": 2000, "renorm": 2000, "predict": 2000}[kind]
    if ny == 6:
        hi = min(hi, 1200)
    if up_bias == 0:
        hi = min(hi, 900 if kind == "trunc" else 400)
    m = int(round(math.exp(rng.uniform(math.log(24), math.log(hi)))))
    split = kind in ("hpsi", "lanczos") and rng.random() < 0.5
    n = nx * ny
    holes = 0 if up_bias == 0 else 2 * max(1, int(round(n * rng.choice([1 / 12, 1 / 10, 1 / 8, 1 / 6]) / 2)))
    return _case(None, kind, nx, ny, m, holes, "split" if split else "fp64", rng.choice([5, 5, 6, 7]) if split else 0,
                 up_bias, rng.choice([0.0, -0.2]), rng.randint(-ny, ny) if nx >= 8 else 0, rng.randint(0, 1),
                 rng.choice([2e-5, 6e-4, 2e-2]) if kind == "lanczos" else 0.0,
                 round(rng.uniform(0.8, 2.6), 2) if kind == "trunc" else 2.2)


# ------------------------------------------------------------------ the inputs
def _lengths(case):
    n = case["nx"] * case["ny"]
    sys_len = n // 2 - 1 + case["shift"]
    return sys_len, n - 2 - sys_len


def _sectors(case, length):
    n = case["nx"] * case["ny"]
    electrons = n - case["holes"] if case["up_bias"] else 0
    return synth.block_sectors(case["m"], electrons * length / n, case["up_bias"], sigma_n=case["sigma"])


def _geometry(case):
    return Geometry(case["nx"], case["ny"], t=1.0, J=1.0 / 3.0, t2=case["t2"], esite=-0.7, up_bias=case["up_bias"])


def _total(case):
    return case["nx"] * case["ny"] - case["holes"] if case["up_bias"] else 0


def _superblock(case, seed):
    sys_len, env_len = _lengths(case)
    electrons = case["nx"] * case["ny"] - case["holes"] if case["up_bias"] else 0
    return synth.make_superblock(case["nx"], case["ny"], sys_len, env_len, case["m"], electrons, seed,
                                 up_bias=case["up_bias"], t2=case["t2"], sigma_n=case["sigma"])


def _graded(sectors, rng):
    """A wavefunction in the bases of a running sweep: block states in order of growing weight (the truncation
    returns them so), amplitudes over two decades on each side."""
    parts = []
    for s in sectors:
        a = np.exp(-math.log(1e2) * (1 - np.arange(s.sys_dim) / s.sys_dim))
        b = np.exp(-math.log(1e2) * (1 - np.arange(s.env_dim) / s.env_dim))
        parts.append((b[:, None] * rng.standard_normal((s.env_dim, s.sys_dim)) * a[None, :]).reshape(-1))
    x = np.concatenate(parts)
    return x / np.linalg.norm(x)


def _schmidt(sectors, rng):
    """A wavefunction of given Schmidt weights in random bases: every sector's singular values fall over two
    decades, the sectors' own scales differ a little (the kept states per sector are those of the sector table)."""
    parts = []
    for i, s in enumerate(sectors):
        k = min(s.sys_dim, s.env_dim)
        u = np.linalg.qr(rng.standard_normal((s.sys_dim, k)))[0]
        v = np.linalg.qr(rng.standard_normal((s.env_dim, k)))[0]
        w = (1 + 0.3 * (i * 0.6180339887498949 % 1)) * np.exp(-math.log(1e2) * np.arange(k) / k)
        parts.append(((v * w) @ u.T).reshape(-1))
    x = np.concatenate(parts)
    return x / np.linalg.norm(x)


def _kept_sectors(trun):
    return [(s.num_up, s.num_down, s.mat.shape[1]) for s in trun.subs]


@lru_cache(maxsize=None)
def _bases(nx, ny, m, holes, up_bias, shift, sigma):
    case = dict(nx=nx, ny=ny, m=m, holes=holes, up_bias=up_bias, shift=shift, sigma=sigma)
    sys_len, env_len = _lengths(case)
    site = synth.site_sectors(up_bias)
    sbs = synth.get_basis(_sectors(case, sys_len), site, sys_len + 1)
    ebs = synth.get_basis(_sectors(case, env_len), site, env_len + 1)
    return sbs, ebs, synth.get_super_basis(sbs, ebs, _total(case), 0)


def _case_bases(case):
    return _bases(case["nx"], case["ny"], case["m"], case["holes"], case["up_bias"], case["shift"], case["sigma"])


def _inputs(case, seed):
    """The numbers a call works on, as host arrays: made from the seed alone."""
    kind = case["kind"]
    if kind in ("hpsi", "lanczos"):
        return _superblock(case, seed)
    rng = np.random.default_rng(seed)
    sys_len, env_len = _lengths(case)
    if kind == "trunc":
        secs = _case_bases(case)[2]
        return structs.Wave(sys_len + 1, env_len + 1, secs, _schmidt(secs, rng))
    if kind == "renorm":
        geo = _geometry(case)
        lat = geo.lattice(sys_len, env_len)
        length = env_len if case["side"] else sys_len
        secs = _sectors(case, length)
        ham, sets = synth.make_ops(secs, length, case["up_bias"], int(geo.nleg11[length - 1]), rng)
        basis = synth.get_basis(secs, synth.site_sectors(case["up_bias"]), length + 1)
        return lat, structs.Model(length, ham, sets), basis, synth.random_trun(basis, case["m"], rng)
    # prediction, left to right or right to left: the block that grows, its truncation just made; the block that
    # shrinks, with the truncation it was once built by
    site = synth.site_sectors(case["up_bias"])
    grow_len, shrink_len = (sys_len, env_len) if case["side"] == 0 else (env_len, sys_len)
    grow_bs = synth.get_basis(_sectors(case, grow_len), site, grow_len + 1)
    u = synth.random_trun(grow_bs, case["m"], rng)
    new_grow_bs = synth.get_basis(_kept_sectors(u), site, grow_len + 2)
    new_shrink_bs = synth.get_basis(_sectors(case, shrink_len - 1), site, shrink_len)
    v = synth.random_trun(new_shrink_bs, case["m"], rng)
    shrink_bs = synth.get_basis(_kept_sectors(v), site, shrink_len + 1)
    total = _total(case)
    if case["side"] == 0:
        old = synth.get_super_basis(grow_bs, shrink_bs, total, 0)
        new = synth.get_super_basis(new_grow_bs, new_shrink_bs, total, 0)
        lens = (sys_len + 1, env_len + 1), (sys_len + 2, env_len)
    else:
        old = synth.get_super_basis(shrink_bs, grow_bs, total, 0)
        new = synth.get_super_basis(new_shrink_bs, new_grow_bs, total, 0)
        lens = (sys_len + 1, env_len + 1), (sys_len, env_len + 2)
    wave = structs.Wave(*lens[0], old, _graded(old, rng))
    return wave, new, lens[1], u, v, new_grow_bs, shrink_bs


# ------------------------------------------------------------------ what a program holds
_CTX = {}


def _context(prec, slices):
    """The program's one context of this precision."""
    if (prec, slices) not in _CTX:
        ctx = lib.Context(0)
        ctx.use_host_pool(True)
        if prec == "split":
            ctx.set_precision(lib.TJ_PREC_OZAKI, slices)
        _CTX[prec, slices] = ctx
    return _CTX[prec, slices]


def _pooled(x):
    a = lib.HOST_POOL.get(max(x.size, 1))
    a[:x.size] = x
    return a


def _pool_wave(w):
    return structs.Wave(w.sys_len, w.env_len, w.sectors, _pooled(w.data))


def _flat_subs(subs, data, off):
    table = (structs.TjBlockSub * max(len(subs), 1))()
    for i, s in enumerate(subs):
        r, c = s.mat.shape
        table[i] = structs.TjBlockSub(s.num_up, s.num_down, s.down_dif, r, c, 0, off)
        data[off:off + r * c] = s.mat.reshape(-1, order="F")
        off += r * c
    return table, off


def _pool_model(m):
    """The model as the library returns it: all blocks in one array of the host pool."""
    blocks = [m.ham] + [getattr(s, k) for s in m.sub for k in structs.OPS]
    data = lib.HOST_POOL.get(max(1, sum(s.mat.size for b in blocks for s in b.subs)))
    keep, cs, off = [data], [], 0
    for b in blocks:
        table, off = _flat_subs(b.subs, data, off)
        keep.append(table)
        cs.append(structs.TjBlock(b.len, len(b.subs), b.dim, b.up_dif, b.down_dif, 0,
                                  C.cast(table, C.POINTER(structs.TjBlockSub)),
                                  data.ctypes.data_as(C.POINTER(C.c_double))))
    sets = (structs.TjBlockSet * max(len(m.sub), 1))()
    for i in range(len(m.sub)):
        sets[i] = structs.TjBlockSet(*cs[1 + 5 * i:6 + 5 * i])
    keep.append(sets)
    c = structs.TjModel(m.len, len(m.sub), cs[0], C.cast(sets, C.POINTER(structs.TjBlockSet)))
    return structs.model_from_c(c, data, keep=keep)


def _pool_trun(b):
    """The truncation operator as the library returns it."""
    data = lib.HOST_POOL.get(max(1, sum(s.mat.size for s in b.subs)))
    table, off = _flat_subs(b.subs, data, 0)
    r = structs.TjTruncResult()
    r.num, r.data_len = len(b.subs), off
    r.sub = C.cast(table, C.POINTER(structs.TjBlockSub))
    r.data = data.ctypes.data_as(C.POINTER(C.c_double))
    return structs.block_from_c_result(r, b.len, table, data)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": dict(case)}
    x = _inputs(case, seed)
    if kind in ("hpsi", "lanczos"):
        state["sb"] = x
        x.sys, x.env = _pool_model(x.sys), _pool_model(x.env)
        x.wave = _pool_wave(x.wave)
        state["packed"] = lib.pack_superblock(x)
        state["out"] = x.wave.like(lib.HOST_POOL.get(max(x.wave.dim, 1)))
        if kind == "hpsi":   # a solve's plan stays with its context
            state["ctx"] = ctx = lib.Context(0)
            if case["prec"] == "split":
                ctx.set_precision(lib.TJ_PREC_OZAKI, case["slices"])
            return state
    elif kind == "trunc":
        state["wave"] = _pool_wave(x)
        state["kept"] = (3 * case["m"] // 4, case["m"])
    elif kind == "renorm":
        lat, pre, basis, trun = x
        state["args"] = (lat, case["side"], 0 if case["side"] == 0 else _lengths(case)[0] + 1, _pool_model(pre), basis,
                         _pool_trun(trun))
    else:
        wave, new, lens, u, v, new_grow_bs, shrink_bs = x
        u, v = _pool_trun(u), _pool_trun(v)
        order = (new_grow_bs, shrink_bs, u, v) if case["side"] == 0 else (shrink_bs, new_grow_bs, v, u)
        new_wave = structs.Wave(*lens, new, lib.HOST_POOL.get(max(1, sum(s.sys_dim * s.env_dim for s in new))))
        state["args"] = (case["side"],) + order + (_pool_wave(wave), new_wave)
    state["ctx"] = _context(case["prec"], case["slices"])
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "hpsi":
        sb, out = state["sb"], state["out"]
        ps, pe, bs, be = state["packed"]
        if lib.lib().tj_model_wave(ctx.h, C.byref(sb.lat.c), C.byref(ps.c), C.byref(pe.c), C.byref(bs.c),
                                   C.byref(be.c), C.byref(sb.wave.c), C.byref(out.c)):
            raise RuntimeError(lib.lib().tj_last_error().decode())
        return out.data
    if kind == "lanczos":
        sb, out = state["sb"], state["out"]
        out.data[:] = sb.wave.data   # the predicted start vector, overwritten by the Ritz vector
        ctx.step_begin()
        e, iters, w = ctx.lanczos_memo_new(sb, case["lanzero"], start=out, packed=state["packed"], in_place=True)
        return {"energy": e, "iters": iters, "ritz": w.data}
    if kind == "trunc":
        r, block = ctx.truncation(state["wave"], case["side"], state["kept"][0], state["kept"][1], 1e-18)
        return {"kept": r.num_state, "weights": np.array([r.trunc_err, r.entropy1, r.entropy2, r.entropys]),
                "operator": block.pack().data}
    if kind == "renorm":
        return ctx.get_hamiltonian(*state["args"]).pack().data
    return ctx.wave_trans(*state["args"]).data


# ------------------------------------------------------------------ recoupling
@lru_cache(maxsize=None)
def _w6j(a, b, c, d, e, f):
    """Wigner 6j symbol {a b c; d e f} of doubled spins, by Racah's sum in exact integers."""
    def tri(x, y, z):
        return abs(x - y) <= z <= x + y and (x + y + z) % 2 == 0
    if not (tri(a, b, c) and tri(a, e, f) and tri(d, b, f) and tri(d, e, c)):
        return 0.0
    g = math.factorial

    def delta(x, y, z):
        return g((x + y - z) // 2) * g((x - y + z) // 2) * g((-x + y + z) // 2), g((x + y + z) // 2 + 1)
    num = den = 1
    for t in ((a, b, c), (a, e, f), (d, b, f), (d, e, c)):
        p, q = delta(*t)
        num, den = num * p, den * q
    lo = [(a + b + c) // 2, (a + e + f) // 2, (d + b + f) // 2, (d + e + c) // 2]
    hi = [(a + b + d + e) // 2, (b + c + e + f) // 2, (c + a + f + d) // 2]
    s, scale = 0, 1
    for k in lo:
        scale *= g(max(hi) - k)
    for k in hi:
        scale *= g(k)
    for t in range(max(lo), min(hi) + 1):
        w = 1
        for k in lo:
            w *= g(t - k)
        for k in hi:
            w *= g(k - t)
        s += (-1) ** t * (g(t + 1) * scale // w if (g(t + 1) * scale) % w == 0 else g(t + 1) * scale / w)
    return float(s) / scale * math.sqrt(num / den)


def _site_ops(ub):
    """Reduced matrix elements of the one-site operators: {kind: (charge, rank, {label: [(label', value)]})}."""
    e, o = (0, 0), (ub, 1)
    return {"eu": (ub, 1, {e: [(o, -math.sqrt(2))]}), "ed": (-ub, 1, {o: [(e, -math.sqrt(2))]}),
            "sd": (0, 2, {o: [(o, math.sqrt(1.5))]}), "sn": (0, 0, {o: [(o, math.sqrt(2))]})}


_FIELD = {"eu": "elec_up", "ed": "elec_down", "sd": "spin_sd", "sn": "num_sn"}


def _moves(basis, charge, rank, mover, targets):
    """Matrix elements of a tensor operator that acts on one part ("block" or "site") of an enlarged basis:
    {(map, sub): [(map', sub', part label, part label', recoupling factor)]}; targets(label) lists the part's
    labels it reaches."""
    where = {}
    for x, mp in enumerate(basis.maps):
        for q, s in enumerate(mp.subs):
            where[mp.new_num_up, mp.new_num_down, s[2], s[3], s[4], s[5]] = (x, q)
    out = {}
    for x, mp in enumerate(basis.maps):
        su, sd = mp.new_num_up, mp.new_num_down
        for q, s in enumerate(mp.subs):
            bl, st = (s[2], s[3]), (s[4], s[5])
            part = bl if mover == "block" else st
            for to in targets(part):
                for nd in range(abs(sd - rank), sd + rank + 1, 2):
                    nb, ns = (to, st) if mover == "block" else (bl, to)
                    at = where.get((su + charge, nd) + nb + ns)
                    if at is None:
                        continue
                    if rank == 0:       # closed form
                        w, ph = 1 / math.sqrt((1 + sd) * (1 + part[1])), 0
                    elif mover == "block":
                        w, ph = _w6j(nd, rank, sd, bl[1], st[1], to[1]), to[1] + st[1] + sd + rank
                    else:
                        w, ph = _w6j(nd, rank, sd, st[1], bl[1], to[1]), bl[1] + st[1] + nd + rank
                    if w:
                        out.setdefault((x, q), []).append((at[0], at[1], part, to, w * (-1) ** (ph // 2)))
    return out


def _reach(labels, charge, rank):
    """Block labels an operator reaches from each (rank 2 vanishes between singlets)."""
    have = set(labels)

    def f(part):
        return [(part[0] + charge, part[1] + dd) for dd in range(-rank, rank + 1, 2)
                if (part[0] + charge, part[1] + dd) in have and not (rank == 2 and dd == 0 and part[1] == 0)]
    return f


def _bonds(lat, sys_len, env_len):
    """Couplings of the superblock: [(where, slot, where, slot, {"eu", "sd", "sn": coefficient})], `where` one of
    block / site of the system (L) or environment (R) side."""
    ns1, nt = lat.num_site + 1, lat.neibt
    neib = lambda i, k: int(lat.neib[k * ns1 + i])          # noqa: E731
    inb1 = lambda i, j: int(lat.inb1[j * ns1 + i])          # noqa: E731
    side = lambda j: int(lat.nposi[lat.nposi_dm[j]])        # noqa: E731
    coup = lambda k, i: {"eu": lat.jt[i * nt + k], "sd": lat.jd[i * nt + k], "sn": lat.jn[k]}   # noqa: E731
    es = int(lat.nposi_lat[sys_len + 1]), int(lat.nposi_lat[sys_len + env_len + 2])
    out = []
    ii = int(lat.neiba[es[1] * ns1 + es[0]])
    if ii:
        out.append(("Ls", 0, "Rs", 0, coup(ii - 1, es[0])))
    for here, lj in (("Ls", es[0]), ("Rs", es[1])):
        for k in range(nt):
            ib = neib(lj, k)
            if side(ib) == 3:
                out.append((here, 0, "Rb", inb1(int(lat.nposi_dm[ib]) - sys_len - 1, env_len) - 1, coup(k, lj)))
            if side(ib) == 1:
                out.append(("Lb", inb1(int(lat.nposi_dm[ib]), sys_len) - 1, here, 0, coup(k, lj)))
    for i in range(1, sys_len + 1):
        for k in range(nt):
            ib = neib(i, k)
            if side(ib) == 3:
                out.append(("Lb", inb1(i, sys_len) - 1, "Rb", inb1(int(lat.nposi_dm[ib]) - sys_len - 1, env_len) - 1,
                            coup(k, i)))
    return out, es


def _inner(basis, charge, rank, sop, labels):
    """Scalar product of a block operator with the site operator inside one enlarged basis:
    [(map, sub, sub', block label, block label', factor)] (factors of the reduced matrix elements)."""
    out = []
    back = {}
    for a, tos in sop[2].items():
        for b, v in tos:
            back.setdefault(b, []).append((a, v))
    reach = _reach(labels, charge, rank)
    for x, mp in enumerate(basis.maps):
        sd = mp.new_num_down
        subs = {(s[2], s[3], s[4], s[5]): q for q, s in enumerate(mp.subs)}
        for q, s in enumerate(mp.subs):
            bl, st = (s[2], s[3]), (s[4], s[5])
            for to in reach(bl):
                for ns, v in back.get(st, []):
                    p = subs.get(to + ns)
                    if p is None:
                        continue
                    if rank == 0:
                        w = 1 / math.sqrt((1 + bl[1]) * (1 + st[1]))
                    else:
                        w = _w6j(to[1], bl[1], rank, st[1], ns[1], sd) * (-1) ** ((bl[1] + ns[1] + rank + sd) // 2)
                    if w:
                        out.append((x, q, p, bl, to, w * v / math.sqrt(1 + rank)))
    return out


def _hpsi_terms(sbs, ebs, secs, lat, sys_len, env_len, ub):
    """H*psi as a list of (out sector, sub, sub, in sector, sub, sub, coefficient, left factor, right factor);
    a factor is None or (side, slot, kind, block label, block label', transposed): out += c A X B^T."""
    ops = _site_ops(ub)
    bonds, es = _bonds(lat, sys_len, env_len)
    lmap = {(m.new_num_up, m.new_num_down): x for x, m in enumerate(sbs.maps)}
    rmap = {(m.new_num_up, m.new_num_down): y for y, m in enumerate(ebs.maps)}
    sec = {(lmap[s.sys_num_up, s.sys_num_down], rmap[s.env_num_up, s.env_num_down]): i for i, s in enumerate(secs)}
    llab = [(s[2], s[3]) for m in sbs.maps for s in m.subs]
    rlab = [(s[2], s[3]) for m in ebs.maps for s in m.subs]
    terms = []
    # block Hamiltonians, site energies
    for (x, y), i in sec.items():
        for q, s in enumerate(sbs.maps[x].subs):
            for p, e in enumerate(ebs.maps[y].subs):
                terms.append((i, q, p, i, q, p, 1 / math.sqrt(1 + s[3]), ("L", -1, "ham", (s[2], s[3]), (s[2], s[3]), 0), None))
                terms.append((i, q, p, i, q, p, 1 / math.sqrt(1 + e[3]), None, ("R", -1, "ham", (e[2], e[3]), (e[2], e[3]), 0)))
                d = lat.esite[es[0]] * (s[5] == 1) + lat.esite[es[1]] * (e[5] == 1)
                if d:
                    terms.append((i, q, p, i, q, p, d, None, None))
    tables = {}
    for wa, sa, wb, sb, coup in bonds:
        for kind, coef in coup.items():
            if coef == 0.0:
                continue
            charge, rank, _ = ops[kind]
            if wa[0] == wb[0]:                              # block and site of one side
                side, basis, lab = ("L", sbs, llab) if wa[0] == "L" else ("R", ebs, rlab)
                slot = sa if wa[1] == "b" else sb
                key = ("in", side, kind)
                if key not in tables:
                    tables[key] = _inner(basis, charge, rank, ops[kind], lab)
                for x, q, p, bl, to, w in tables[key]:
                    if rank == 1:   # the fermion passes the block (L) or, reordered, the emptied site (R)
                        w = w * ((-1) ** bl[1] if side == "L" else 1)
                    f, ft = (side, slot, kind, bl, to, 0), (side, slot, kind, bl, to, 1)
                    for (xs, ys), i in sec.items():
                        if (xs if side == "L" else ys) != x:
                            continue
                        for r in range(len((ebs.maps[ys] if side == "L" else sbs.maps[xs]).subs)):
                            a, b = ((q, r), (p, r)) if side == "L" else ((r, q), (r, p))
                            terms.append((i, *b, i, *a, coef * w) + ((f, None) if side == "L" else (None, f)))
                            if rank == 1:
                                terms.append((i, *a, i, *b, coef * w) + ((ft, None) if side == "L" else (None, ft)))
                continue
            rkind = {"eu": "ed"}.get(kind, kind)             # the other side takes the charge back
            for key, basis, lab, knd in (((wa, kind), sbs, llab, kind), ((wb, rkind), ebs, rlab, rkind)):
                if key not in tables:
                    ch, rk, vals = ops[knd]
                    to = _reach(lab, ch, rk) if key[0][1] == "b" else (lambda part, v=vals: [t for t, _ in v.get(part, [])])
                    tables[key] = _moves(basis, ch, rk, "block" if key[0][1] == "b" else "site", to)
            left, right = tables[wa, kind], tables[wb, rkind]
            val = {k: {(a, b): v for a, t in ops[k][2].items() for b, v in t} for k in (kind, rkind)}
            for (x, y), i in sec.items():
                sd, ed = sbs.maps[x].new_num_down, ebs.maps[y].new_num_down
                for q, s in enumerate(sbs.maps[x].subs):
                    for x2, q2, la, lb, wl in left.get((x, q), []):
                        for p, e in enumerate(ebs.maps[y].subs):
                            for y2, p2, ra, rb, wr in right.get((y, p), []):
                                if sbs.maps[x2].new_num_down != ebs.maps[y2].new_num_down or (x2, y2) not in sec:
                                    continue
                                ned = ebs.maps[y2].new_num_down
                                c = coef * wl * wr * math.sqrt((1 + ned) * (1 + ed) / (1 + rank))
                                if rank == 1:
                                    c *= (-1) ** ((0 if wa[1] == "b" else s[3]) + sd + (e[5] if wb[1] == "b" else 0))
                                fl = fr = None
                                if wa[1] == "b":
                                    fl = ("L", sa, kind, la, lb)
                                else:
                                    c *= val[kind][la, lb]
                                if wb[1] == "b":
                                    fr = ("R", sb, rkind, ra, rb)
                                else:
                                    c *= val[rkind][ra, rb]
                                j = sec[x2, y2]
                                terms.append((j, q2, p2, i, q, p, c, fl and fl + (0,), fr and fr + (0,)))
                                if rank == 1:
                                    terms.append((i, q, p, j, q2, p2, c, fl and fl + (1,), fr and fr + (1,)))
    return terms


def _term_cost(case):
    """(flops, bytes) one H*psi cannot do without: every distinct product once, every operator and psi once."""
    sbs, ebs, secs = _case_bases(case)
    sys_len, env_len = _lengths(case)
    geo = _geometry(case)
    lat = geo.lattice(sys_len, env_len)
    terms = _hpsi_terms(sbs, ebs, secs, lat, sys_len, env_len, case["up_bias"])
    maps = {(m.new_num_up, m.new_num_down): m for m in sbs.maps}, {(m.new_num_up, m.new_num_down): m for m in ebs.maps}
    dl = lambda i, q: maps[0][secs[i].sys_num_up, secs[i].sys_num_down].subs[q][1]      # noqa: E731
    dr = lambda i, p: maps[1][secs[i].env_num_up, secs[i].env_num_down].subs[p][1]      # noqa: E731
    flops, prods, second, used = 0.0, set(), {}, {}
    for j, q2, p2, i, q, p, c, fl, fr in terms:
        M, N, K1, K2 = dl(j, q2), dr(j, p2), dl(i, q), dr(i, p)
        for f, n in ((fl, M * K1), (fr, N * K2)):
            if f:
                used[f[:-1]] = n
        if fl and fr:
            if (fl, i, q, p) not in prods:
                prods.add((fl, i, q, p))
                flops += 2.0 * M * K1 * K2
            second[(fl, j, q2, p2, i, q, p, fr[0], fr[2:])] = 2.0 * M * K2 * N   # the right operators of a site pre-summed
        elif fl or fr:
            f = fl or fr
            second[(f[0], f[2:], j, q2, p2, i, q, p)] = 2.0 * M * N * (K1 if fl else K2)
    dim = sum(s.sys_dim * s.env_dim for s in secs)
    return flops + sum(second.values()), 8.0 * (sum(used.values()) + 2 * dim), dim


@lru_cache(maxsize=None)
def _work(key):
    case = dict(key)
    kind, m = case["kind"], case["m"]
    if kind in ("hpsi", "lanczos"):
        flops, nbytes, dim = _term_cost(case)
        if kind == "hpsi":
            return nbytes, flops
        # iterations of such a solve, each with its vector algebra: every earlier vector read twice
        it = {2e-5: 60, 6e-4: 45, 2e-2: 28}.get(case["lanzero"], 60)
        return nbytes + it * 8.0 * dim * (6 + it), it * (flops + 2.0 * dim * (6 + it))
    if kind == "trunc":
        secs = _case_bases(case)[2]
        dims = [(s.sys_dim, s.env_dim) if case["side"] == 0 else (s.env_dim, s.sys_dim) for s in secs]
        kept = m / max(1, sum(d for d, _ in dims))
        flops = sum(d * d * k + 4 / 3 * d ** 3 + 2 * (kept * d) * d * d + 2 * (kept * d) ** 2 * d for d, k in dims)
        return 8.0 * sum(d * k + kept * d * d for d, k in dims), flops
    sys_len, env_len = _lengths(case)
    site = synth.site_sectors(case["up_bias"])
    if kind == "renorm":
        geo = _geometry(case)
        length = env_len if case["side"] else sys_len
        secs = _sectors(case, length)
        basis = synth.get_basis(secs, site, length + 1)
        kept = {(b.new_num_up, b.new_num_down): max(1, min(b.dim, round(m * b.dim / basis.dim))) for b in basis.maps}
        dims = {(s[0], s[1]): s[2] for s in secs}
        flops, nbytes = 0.0, 8.0 * sum(kept[b.new_num_up, b.new_num_down] * b.dim for b in basis.maps)
        ub = case["up_bias"]
        n0, n1 = int(geo.nleg11[length - 1]), int(geo.nleg11[length])
        for charge, rank, count in ((0, 0, 1), (ub, 1, n1), (-ub, 1, n1), (0, 2, n1), (0, 0, n1)):
            reach = _reach(dims, charge, rank)
            per = 8.0 * sum(dims[a] * dims[b] for a in dims for b in reach(a))
            nbytes += per * (1 if count == 1 else n0)
            for (x, q), tos in _moves(basis, charge, rank, "block", reach).items():
                r = kept[basis.maps[x].new_num_up, basis.maps[x].new_num_down]
                for x2, _, a, b, _ in tos:
                    l = kept[basis.maps[x2].new_num_up, basis.maps[x2].new_num_down]
                    flops += count * (2.0 * min(dims[b] * dims[a] * r, l * dims[b] * dims[a]) + 2.0 * l * r * min(dims[a], dims[b]))
            nbytes += count * 8.0 * sum(kept[a] * kept[b] for a in kept for b in _reach(kept, charge, rank)(a))
        return nbytes, flops
    old, new, u, v, flops = _predict_shape(case)
    return 8.0 * (old + new + u + v), flops


def _predict_shape(case):
    sys_len, env_len = _lengths(case)
    site = synth.site_sectors(case["up_bias"])
    g, s = (sys_len, env_len) if case["side"] == 0 else (env_len, sys_len)

    def kept(basis):
        return [(b.new_num_up, b.new_num_down, max(1, min(b.dim, int(round(case["m"] * b.dim / basis.dim))))) for b in basis.maps]
    gb = synth.get_basis(_sectors(case, g), site, g + 1)
    ng = synth.get_basis(kept(gb), site, g + 2)
    ns = synth.get_basis(_sectors(case, s - 1), site, s)
    sb = synth.get_basis(kept(ns), site, s + 1)
    size = lambda a, b: sum(w.sys_dim * w.env_dim for w in synth.get_super_basis(a, b, _total(case), 0))   # noqa: E731
    ku, kv = {k[:2]: k[2] for k in kept(gb)}, {k[:2]: k[2] for k in kept(ns)}
    du, dv = ({(b.new_num_up, b.new_num_down): b.dim for b in x.maps} for x in (gb, ns))
    flops = 0.0
    for w in synth.get_super_basis(gb, sb, _total(case), 0):
        a = (w.sys_num_up, w.sys_num_down)
        flops += 2.0 * ku[a] * du[a] * w.env_dim            # U^T psi, then V per sub-block of the shrinking side
        b = next(t for t in sb.maps if (t.new_num_up, t.new_num_down) == (w.env_num_up, w.env_num_down))
        for t in b.subs:
            flops += 2.0 * ku[a] * kv[t[2], t[3]] * dv[t[2], t[3]]
    return size(gb, sb), size(ng, ns), sum(ku[k] * du[k] for k in ku), sum(kv[k] * dv[k] for k in kv), flops


def work(case):
    b, f = _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_DEV)


def _mats(block):
    return {((s.num_up, s.num_down), (s.num_up + block.up_dif, s.num_down + s.down_dif)): _t(s.mat) for s in block.subs}


def _views(data, secs):
    """Per sector the (sys_dim, env_dim) view of a flat vector (columns contiguous)."""
    out, off = [], 0
    for s in secs:
        n = s.sys_dim * s.env_dim
        out.append(data[off:off + n].view(s.env_dim, s.sys_dim).t())
        off += n
    return out


def _hpsi_operator(case, sb):
    """psi -> H psi on flat torch vectors."""
    sys_len, env_len = sb.sys.len, sb.env.len
    secs = sb.wave.sectors
    mats = {}
    for side, model in (("L", sb.sys), ("R", sb.env)):
        mats[side, -1, "ham"] = _mats(model.ham)
        for i, bs in enumerate(model.sub):
            for k, f in _FIELD.items():
                mats[side, i, k] = _mats(getattr(bs, f))
    terms = _hpsi_terms(sb.sys_bs, sb.env_bs, secs, sb.lat, sys_len, env_len, case["up_bias"])
    lm = {(b.new_num_up, b.new_num_down): b for b in sb.sys_bs.maps}
    rm = {(b.new_num_up, b.new_num_down): b for b in sb.env_bs.maps}
    win = []
    for s in secs:
        win.append(([slice(t[0], t[0] + t[1]) for t in lm[s.sys_num_up, s.sys_num_down].subs],
                    [slice(t[0], t[0] + t[1]) for t in rm[s.env_num_up, s.env_num_down].subs]))
    # terms of one output window and input window and left factor share their product; right factors are summed
    grouped, rsum = {}, {}
    for j, q2, p2, i, q, p, c, fl, fr in terms:
        g = grouped.setdefault((j, q2, p2, i, q, p, fl), {})
        g[fr] = g.get(fr, 0.0) + c
    plan, scalar, left = [], {}, {}
    for (j, q2, p2, i, q, p, fl), g in grouped.items():
        for fr, c in g.items():
            if fl is None and fr is None:
                scalar[j, q2, p2, i, q, p] = scalar.get((j, q2, p2, i, q, p), 0.0) + c
            elif fl is None or fr is None:      # one-sided: sum the operators of all slots
                f = fl or fr
                op = mats[f[:3]][f[3], f[4]]
                key = (j, q2, p2, i, q, p, fl is None)
                left.setdefault(key, []).append((c, op.t() if f[5] else op))
        two = tuple(sorted(((fr, c) for fr, c in g.items() if fl is not None and fr is not None), key=repr))
        if two:
            if two not in rsum:
                rsum[two] = sum(c * (mats[f[:3]][f[3], f[4]].t() if f[5] else mats[f[:3]][f[3], f[4]]) for f, c in two).t()
            a = mats[fl[:3]][fl[3], fl[4]]
            plan.append((j, q2, p2, i, q, p, fl, a.t() if fl[5] else a, rsum[two]))
    plan.sort(key=lambda t: (t[3], t[4], t[5], repr(t[6])))
    ones = [(k, sum(c * o for c, o in v)) for k, v in left.items()]

    def apply(x):
        y = torch.zeros_like(x)
        X, Y = _views(x, secs), _views(y, secs)
        cut = lambda V, i, q, p: V[i][win[i][0][q], win[i][1][p]]      # noqa: E731
        for (j, q2, p2, i, q, p), c in scalar.items():
            cut(Y, j, q2, p2).add_(cut(X, i, q, p), alpha=c)
        for (j, q2, p2, i, q, p, right), op in ones:
            w = cut(X, i, q, p)
            cut(Y, j, q2, p2).add_(w @ op.t() if right else op @ w)
        last, prod = None, None
        for j, q2, p2, i, q, p, fl, a, b in plan:
            if (i, q, p, fl) != last:
                last, prod = (i, q, p, fl), a @ cut(X, i, q, p)
            cut(Y, j, q2, p2).add_(prod @ b)
        return y
    return apply, len(plan) * 2 + len(ones)


def _exact_lanczos(apply, start, lanzero):
    v = [start / start.norm()]
    w = apply(v[0])
    alpha, beta = [float(v[0] @ w)], []
    ritz = alpha[0]
    while len(v) < 110:
        n = len(v)
        w = w - alpha[-1] * v[-1]
        if n >= 2:
            w = w - beta[-1] * v[-2]
        b = float(w.norm())
        if abs(b) <= lanzero:
            break
        w = w / b
        V = torch.stack(v)
        w = w - V.t() @ (V @ w)
        w = w / w.norm()
        v.append(w)
        beta.append(b)
        w = apply(v[-1])
        alpha.append(float(v[-1] @ w))
        T = np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1)
        new = float(np.linalg.eigvalsh(T)[0])
        done = abs(new - ritz) <= lanzero
        ritz = new
        if done:
            break
    n = len(v)
    ev, z = np.linalg.eigh(np.diag(alpha) + np.diag(beta[:n - 1], 1) + np.diag(beta[:n - 1], -1))
    z = z[:, 0] * (1.0 if z[0, 0] > 0 else -1.0)
    r = torch.stack(v).t() @ _t(z)
    return {"energy": float(ev[0]), "iters": n, "ritz": r / r.norm()}


def _exact_trunc(case, wave, kept_min, kept_max):
    x = _t(wave.data[:wave.dim])
    nrm2 = float(x @ x)
    side, vals, vecs, rows = case["side"], [], [], []
    for s, m in zip(wave.sectors, _views(x, wave.sectors)):
        e, q = torch.linalg.eigh((m @ m.t() if side == 0 else m.t() @ m) / nrm2)
        vals.append(e.cpu().numpy())
        vecs.append(q)
        rows.append((s.sys_num_down if side == 0 else s.env_num_down) + 1)
    val = np.concatenate(vals)
    own = np.concatenate([np.full(len(v), i) for i, v in enumerate(vals)])
    mult = np.array(rows)[own]
    thr = float(np.float32(1e-15))
    order = np.argsort(-val, kind="stable")
    w = val[order] / val.sum()
    n, err = len(val), 0.0
    if len(val) > kept_min:
        n, err = kept_min, float(w[kept_min:].sum())
        while err > 1e-18 and n < len(val):
            n += 1
            err -= w[n - 1]
            if err <= 1e-18 or n >= kept_max:
                break
    ent = lambda p, g: float(-(g[p >= thr] * p[p >= thr] * np.log(p[p >= thr])).sum())      # noqa: E731
    v1 = np.where(val >= thr, val / mult, 0.0)
    count = np.bincount(own[order[:n]], minlength=len(vals))
    parts = []
    for i, q in enumerate(vecs):
        k = int(count[i])
        if k == 0:
            continue
        u = q[:, q.shape[1] - k:]
        top = u.abs().argmax(dim=0)
        u = u * torch.sign(u[top, torch.arange(k, device=u.device)])[None, :]
        parts.append(u.t().reshape(-1))
    return {"kept": n, "weights": np.array([float(w[n:].sum()) if n < len(val) else 0.0,
                                            float(-(mult[v1 > 0] * v1[v1 > 0] * np.log(v1[v1 > 0])).sum()),
                                            ent(val / (val * mult).sum(), mult), ent(w, np.ones_like(w))]),
            "operator": torch.cat(parts)}


def _exact_renorm(case, lat, pre, basis, trun):
    ub, side = case["up_bias"], case["side"]
    length, sys_len = pre.len, _lengths(case)[0]
    ns1, nt = lat.num_site + 1, lat.neibt
    inb1 = lambda i, j: int(lat.inb1[j * ns1 + i])                # noqa: E731
    ops = _site_ops(ub)
    mats = [{k: _mats(getattr(s, f)) for k, f in _FIELD.items()} for s in pre.sub]
    lab = {(s[2], s[3]) for m in basis.maps for s in m.subs}
    U = {(s.num_up, s.num_down): _t(s.mat) for s in trun.subs}
    at = {(m.new_num_up, m.new_num_down): x for x, m in enumerate(basis.maps)}
    cut = [[slice(s[0], s[0] + s[1]) for s in m.subs] for m in basis.maps]
    dim = [m.dim for m in basis.maps]
    zeros = lambda l, r: torch.zeros(dim[l], dim[r], dtype=torch.float64, device=_DEV)      # noqa: E731

    def enlarged(kind, block=None):
        """{(map', map): matrix} of a block operator (given) or of the new site's operator."""
        charge, rank, vals = ops[kind]
        out = {}
        reach = _reach(lab, charge, rank) if block is not None else (lambda part: [t for t, _ in vals.get(part, [])])
        for (x, q), tos in _moves(basis, charge, rank, "block" if block is not None else "site", reach).items():
            s = basis.maps[x].subs[q]
            for x2, q2, a, b, w in tos:
                w *= math.sqrt((1 + basis.maps[x].new_num_down) * (1 + basis.maps[x2].new_num_down))
                if rank == 1 and (side == 1) == (block is not None):
                    w *= (-1) ** (s[5] if block is not None else s[3])
                o = out.setdefault((x2, x), zeros(x2, x))
                if block is not None:
                    o[cut[x2][q2], cut[x][q]] += w * block[a, b]
                else:
                    o[cut[x2][q2], cut[x][q]] += w * dict(vals[a])[b] * torch.eye(s[1], dtype=torch.float64, device=_DEV)
        return out

    ham = {(x, x): zeros(x, x) for x in range(len(basis.maps))}
    h0 = _mats(pre.ham)
    site = length + 1 + (0 if side == 0 else sys_len + 1)
    jl = int(lat.nposi_lat[site]) if side else site
    for x, m in enumerate(basis.maps):
        for q, s in enumerate(m.subs):
            w = ham[x, x][cut[x][q], cut[x][q]]
            w += math.sqrt((1 + m.new_num_down) / (1 + s[3])) * h0[(s[2], s[3]), (s[2], s[3])]
            if s[5] == 1:
                w += lat.esite[jl] * math.sqrt(1 + m.new_num_down) * torch.eye(s[1], dtype=torch.float64, device=_DEV)
    for k in range(nt):
        i = int(lat.neib[k * ns1 + jl])
        i = (int(lat.nposi_dm[i]) - (sys_len + 1)) if side else i
        if not 0 < i <= length or not 0 < inb1(i, length) <= len(pre.sub):
            continue
        for kind, coef in (("eu", lat.jt[jl * nt + k]), ("sd", lat.jd[jl * nt + k]), ("sn", lat.jn[k])):
            if coef == 0.0:
                continue
            charge, rank, _ = ops[kind]
            block = mats[inb1(i, length) - 1][kind]
            for x, q, p, a, b, w in _inner(basis, charge, rank, ops[kind], lab):
                w *= coef * math.sqrt(1 + basis.maps[x].new_num_down)
                if rank == 1 and side == 0:
                    w *= (-1) ** a[1]
                ham[x, x][cut[x][p], cut[x][q]] += w * block[a, b]
                if rank == 1:
                    ham[x, x][cut[x][q], cut[x][p]] += w * block[a, b].t()
    secs = [(s.num_up, s.num_down) for s in trun.subs]
    out = []

    def truncated(op, charge, rank):
        for r in secs:
            for dd in range(-rank, rank + 1, 2):
                l = (r[0] + charge, r[1] + dd)
                if l not in U:
                    continue
                e = op.get((at[l], at[r]))
                y = U[l].t() @ e @ U[r] if e is not None else torch.zeros(U[l].shape[1], U[r].shape[1], dtype=torch.float64, device=_DEV)
                out.append(y.t().reshape(-1))
    truncated(ham, 0, 0)
    slots = {}
    for i in range(1, length + 1):
        if inb1(i, length) <= len(pre.sub) and inb1(i, length + 1) <= int(lat.nleg11[length]):
            slots[inb1(i, length + 1)] = inb1(i, length) - 1
    for j in range(1, int(lat.nleg11[length]) + 1):
        for kind in ("eu", "ed", "sd", "sn"):
            src = slots.get(j) if j != inb1(length + 1, length + 1) else None
            truncated(enlarged(kind, mats[src][kind] if src is not None else None), ops[kind][0], ops[kind][1])
    return torch.cat(out)


def _exact_predict(case, wave, new, u, v, new_grow_bs, shrink_bs):
    U = {(s.num_up, s.num_down): _t(s.mat) for s in u.subs}
    V = {(s.num_up, s.num_down): _t(s.mat) for s in v.subs}
    gm = {(m.new_num_up, m.new_num_down): m for m in new_grow_bs.maps}
    sm = {(m.new_num_up, m.new_num_down): m for m in shrink_bs.maps}
    out = torch.zeros(sum(s.sys_dim * s.env_dim for s in new), dtype=torch.float64, device=_DEV)
    left = case["side"] == 0
    Y = {(s.sys_num_up, s.sys_num_down, s.env_num_up, s.env_num_down): y for s, y in zip(new, _views(out, new))}
    for s, x in zip(wave.sectors, _views(_t(wave.data[:wave.dim]), wave.sectors)):
        g, sh = (s.sys_num_up, s.sys_num_down), (s.env_num_up, s.env_num_down)
        if not left:
            g, sh, x = sh, g, x.t()
        for spos, sdim, bu, bd, stu, std in sm[sh].subs:
            w = U[g].t() @ x[:, spos:spos + sdim] @ V[bu, bd].t()
            for nd in range(abs(g[1] - std), g[1] + std + 1, 2):
                n = (g[0] + stu, nd)
                y = Y.get(n + (bu, bd) if left else (bu, bd) + n)
                if y is None:
                    continue
                p = next(t for t in gm[n].subs if t[2:] == (g[0], g[1], stu, std))
                # psi[(g), (b s) sh; 0] -> psi'[(g s) nd, b; 0]: one 6j symbol with a vanishing spin, closed form
                c = math.sqrt((1 + sh[1]) / (1 + g[1]))
                if left:
                    c *= (-1) ** ((g[1] + std + nd) // 2 + (g[1] + std + bd) // 2 + (std + bd - sh[1]) // 2)
                else:
                    c = math.sqrt((1 + nd) * (1 + sh[1]) / ((1 + g[1]) * (1 + bd)))
                    c *= (-1) ** ((sh[1] + bd + std) // 2 + (bd + std + g[1]) // 2 + (g[1] + std - nd) // 2)
                (y if left else y.t())[p[0]:p[0] + p[1], :] += c * w
    return out / out.norm()


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "hpsi":
        return _hpsi_operator(case, x)[0](_t(x.wave.data[:x.wave.dim]))
    if kind == "lanczos":
        apply, n = _hpsi_operator(case, x)
        if n > 12000:   # some tens of products: over twenty seconds
            return None
        return _exact_lanczos(apply, _t(x.wave.data[:x.wave.dim]), case["lanzero"])
    if kind == "trunc":
        return _exact_trunc(case, x, 3 * case["m"] // 4, case["m"])
    if kind == "renorm":
        return _exact_renorm(case, *x)
    wave, new, _, u, v, new_grow_bs, shrink_bs = x
    return _exact_predict(case, wave, new, u, v, new_grow_bs, shrink_bs)
