"""Instance sets of nothing, and of plans that cannot be enumerated: an error
only where there are rows to write."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def match(sge, eng, b, p, cap, labels=None):
    ph = C.c_void_p()
    sge._check(sge.lib().sge_plan_create(C.byref(b), C.byref(ph)))
    if labels is not None:
        sge._check(sge.lib().sge_plan_set_labels(ph, sge._u32p(np.array(labels, np.uint32))))
    out, rows, e = np.full(max(cap, 1) * p.k, 7, np.uint32), C.c_uint64(99), p.flat()
    st = sge.lib().sge_match_set(eng._h, ph, p.k, p.m, sge._u32p(e), sge._u32p(out), cap, C.byref(rows))
    sge.lib().sge_plan_destroy(ph)
    return sge.STATUS[st], rows.value, out


@pytest.mark.parametrize("cap", [0, 5, 5000])
def test_labeled_and_long_tail_plans(sge, cap):
    tri = sge.PatternGraph.from_edges(3, [(0, 1), (0, 2), (1, 2)])
    star = sge.PatternGraph.from_edges(4, [(0, 1), (0, 2), (0, 3)])
    k4 = sge.PatternGraph.from_edges(4, [(a, b) for a in range(4) for b in range(a + 1, 4)])
    with sge.Engine(sge.gen_chung_lu(200, 700, 2.1, 80, seed=1)) as eng:
        eng.set_labels(np.arange(200) % 2)
        few = sge.plan(tri, eng, labels=[0, 0, 1])
        none = sge.plan(tri, eng, labels=[0, 0, 5])
        n = eng.count([few], labels=[[0, 0, 1]])[1][0]
        assert 5 < n < 5000
        assert match(sge, eng, none, tri, cap, [0, 0, 5])[:2] == ("OK", 0)
        assert match(sge, eng, few, tri, cap, [0, 0, 1])[:2] == ("UNSUPPORTED" if cap > n else "OOM", n)
        long_tail = sge.plan(star, eng, iep=True)
        assert long_tail.tail_len > 1
        s = eng.count([long_tail])[1][0]
        assert match(sge, eng, long_tail, star, cap)[:2] == ("BAD_INPUT" if cap > s else "OOM", s)
    with sge.Engine(sge.DataGraph.from_edges(np.array([(i, i + 1) for i in range(50)]), 51)) as eng:
        assert match(sge, eng, sge.plan(k4, eng, iep=False), k4, cap)[:2] == ("OK", 0)
        assert eng.match_set(k4).shape == (0, 4)


@pytest.mark.parametrize("more", [-1, 1])
def test_rows_are_compared_with_the_count(sge, monkeypatch, more):
    tri = sge.PatternGraph.from_edges(3, [(0, 1), (0, 2), (1, 2)])
    with sge.Engine(sge.gen_chung_lu(200, 700, 2.1, 80, seed=1)) as eng:
        count = eng.count
        rows = len(eng.match_set(tri))

        def wrong(plans, **kw):
            c, inst, st = count(plans, **kw)
            return c, [n + more for n in inst], st
        monkeypatch.setattr(eng, "count", wrong)
        with pytest.raises(sge.SgeError) as e:
            eng.match_set(tri)
        assert e.value.status_name == ("CUDA_ERROR" if more > 0 else "OOM")
        monkeypatch.undo()
        assert len(eng.match_set(tri)) == rows
