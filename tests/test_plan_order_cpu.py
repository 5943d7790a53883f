"""Work items of the grouped GEMM come heaviest first, ties in the order of
their cells, and cover every tile's tasks exactly once."""
import pytest

from grand_sql_tj_b200 import synth
from grand_sql_tj_b200.lib import plan_export


@pytest.mark.parametrize("wl", ["tiny", "small_gc", "cyl4", "ladder16_m256"])
def test_items_sorted_and_complete(wl, product_lib):
    d = plan_export(synth.workload(wl, seed=3))
    for ph in (1, 2):
        n = getattr(d["ex"], "n_items%d" % ph)
        cells, tasks, items = d["cells%d" % ph], d["tasks%d" % ph], list(d["items%d" % ph][:n])
        weight = [1 + sum(tasks[t].K for t in range(i.tb, i.te)) for i in items]
        key = [(-w, i.cell, i.row0, i.col0, i.tb) for w, i in zip(weight, items)]
        assert key == sorted(key)
        seen = {}
        for i in items:
            seen.setdefault((i.cell, i.row0, i.col0), []).append((i.tb, i.te))
        for c in range(getattr(d["ex"], "n_cells%d" % ph)):
            gemm = [t for t in range(cells[c].t_begin, cells[c].t_end) if tasks[t].R.space != 0]
            for r in range(0, cells[c].M, 64):
                for q in range(0, cells[c].N, 64):
                    got = [t for tb, te in sorted(seen.pop((c, r, q))) for t in range(tb, te)]
                    assert got == gemm
        assert not seen
