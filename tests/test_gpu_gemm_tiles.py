"""The grouped FP64 GEMM at the edges of its tiles: row and column counts around
the 8-entry granules and the 64-entry tile, inner dimensions around the groups
of four and the 32-entry steps, operands stored either way with odd leading
dimensions and offsets, cells of more tasks than the 32 a copying warp holds at
a time, and cells split over several work items and summed (reduce).

Tolerance: an entry is a sum of n products of three factors; in FP64, in any
order, its error is below (n + 2) 2^-53 sum |coef L R| (each product rounded
twice, n - 1 additions), checked entry by entry.
"""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from grand_sql_tj_b200 import gg
from grand_sql_tj_b200.structs import TjGgCell, TjGgTerm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(product_lib):
    from grand_sql_tj_b200.lib import Context
    c = Context(0)
    yield c
    c.close()


def _batch(shapes, rng):
    """shapes: (M, N, [K, ...]) per cell; operands at odd places of one pool."""
    pool = rng.standard_normal(1 << 18)
    cells = (TjGgCell * len(shapes))()
    terms, off = [], 0
    for c, (M, N, Ks) in enumerate(shapes):
        t0 = len(terms)
        for K in Ks:
            lt, rt = int(rng.integers(2)), int(rng.integers(2))
            ldl, ldr = (K if lt else M) + int(rng.integers(4)), (N if rt else K) + int(rng.integers(4))
            ll, rl = ldl * (M if lt else K), ldr * (K if rt else N)
            terms.append(TjGgTerm(int(rng.integers(pool.size - ll)), int(rng.integers(pool.size - rl)), ldl, ldr, K, lt, rt,
                                  0, float(rng.uniform(-1, 1))))
        cells[c] = TjGgCell(off, M, N, t0, len(terms))
        off += M * N
    return SimpleNamespace(cells=cells, terms=(TjGgTerm * len(terms))(*terms), pool=pool, out_len=off)


def _check(ctx, b):
    _, out, _, _ = ctx.grouped_gemm_bench(b, 0, reps=1)
    ref = gg.reference(b)
    mag = gg.reference(SimpleNamespace(cells=b.cells, pool=np.abs(b.pool), terms=[
        TjGgTerm(*[getattr(t, f) for f, _ in TjGgTerm._fields_[:-1]], abs(t.coef)) for t in b.terms]))
    for c in ref:
        n = sum(b.terms[t].K for t in range(b.cells[c].t_begin, b.cells[c].t_end))
        # the reference is such a sum too
        bound = 2 * (n + 2) * 2.0 ** -53 * mag[c]
        assert np.all(np.abs(gg.cell_view(b, out, c) - ref[c]) <= bound), (c, b.cells[c].M, b.cells[c].N)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 56, 57, 64, 65, 130])
def test_tile_edges(ctx, M):
    rng = np.random.default_rng(M)
    Ks = [1, 3, 4, 5, 13, 28, 29, 31, 32, 33, 36, 64, 67]
    shapes = [(M, N, [Ks[int(k)] for k in rng.integers(len(Ks), size=int(rng.integers(1, 6)))])
              for N in (1, 5, 8, 11, 16, 24, 31, 40, 64, 71, 129)]
    _check(ctx, _batch(shapes, rng))


def test_many_tasks_and_split_cells(ctx):
    rng = np.random.default_rng(5)
    shapes = [(20, 30, [1] * 31), (20, 30, [2] * 32), (9, 70, [5] * 33), (66, 12, [3] * 97), (1, 1, [1] * 200),
              (65, 130, [40] * 60), (64, 64, [31] * 40), (3, 3, [100] * 9)]
    _check(ctx, _batch(shapes, rng))
