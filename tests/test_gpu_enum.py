"""Enumerated instance sets against the CPU oracle's embedding list: three-
vertex patterns (32 roots at a time), the flattened last two levels of longer
ones, lists longer than a warp, hubs at either end of the id order, and an
output buffer that is too small."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = {
    "triangle": (3, [(0, 1), (0, 2), (1, 2)]),
    "wedge": (3, [(0, 1), (1, 2)]),
    "cycle4": (4, [(0, 1), (1, 2), (2, 3), (0, 3)]),
    "star3": (4, [(0, 1), (0, 2), (0, 3)]),
    "k4": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]),
    "house": (5, [(0, 1), (0, 2), (0, 4), (1, 3), (1, 4), (2, 3)]),
    "k5_minus_e": (5, [(a, b) for a in range(5) for b in range(a + 1, 5) if (a, b) != (3, 4)]),
}


def graph(sge, kind, reverse):
    if kind == "chung_lu":
        g = sge.gen_chung_lu(90, 330, 2.1, 60, seed=3)
    else:  # two hubs over a sparse rest: scans of several warps' length
        e = [(0, i) for i in range(2, 80)] + [(1, i) for i in range(2, 80, 2)] + [(i, i + 1) for i in range(2, 79)] + [(0, 1)]
        g = sge.DataGraph.from_edges(np.array(e), 80)
    if reverse:
        g = sge.DataGraph.from_edges(g.num_vertices - 1 - g.edge_array().astype("int64"), g.num_vertices)
    return g


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("kind", ["chung_lu", "hubs"])
@pytest.mark.parametrize("name", list(PATTERNS))
def test_instance_sets_match_the_oracle(sge, oracle, name, kind, reverse):
    k, edges = PATTERNS[name]
    p = sge.PatternGraph.from_edges(k, edges)
    g = graph(sge, kind, reverse)
    perms = (C.c_uint8 * (4096 * k))()
    n = C.c_uint32()
    e = p.flat()
    sge._check(sge.lib().sge_pattern_automorphisms(k, p.m, sge._u32p(e), perms, 4096, C.byref(n)))
    perms = np.array(perms[: n.value * k]).reshape(n.value, k)
    want = oracle.canonical_instances(oracle.list_embeddings(g.offsets, g.nbrs, k, p.edges), perms)
    with sge.Engine(g) as eng:
        for exploration in (False, True):
            got = eng.match_set(p, exploration=exploration)
            assert got.shape == want.shape and np.array_equal(got, want)
        if len(want) > 1:   # a smaller buffer: the status, the true count, and no row past the end
            b = sge.plan(p, eng, iep=False)
            ph = C.c_void_p()
            sge._check(sge.lib().sge_plan_create(C.byref(b), C.byref(ph)))
            out = np.full(len(want) * k, 7, np.uint32)
            rows = C.c_uint64()
            st = sge.lib().sge_match_set(eng._h, ph, k, p.m, sge._u32p(e), sge._u32p(out), len(want) - 1, C.byref(rows))
            sge.lib().sge_plan_destroy(ph)
            assert sge.STATUS[st] == "OOM" and rows.value == len(want) and (out == 7).all()
