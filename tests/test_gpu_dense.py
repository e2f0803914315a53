"""Roots counted on bitsets (csrc/dense.cuh) against the list path and the CPU
oracle.  A run with an explicit list capacity (here the largest degree, which
no list exceeds) keeps every root on lists, so the two paths are compared on
the same plans: one and two words per lane, universes that do not fit, the
three tail modes, both join styles, root samples and degree caps."""
import pytest

pytestmark = pytest.mark.gpu


def rooted(sge, p, stats, **kw):
    import bench
    seq, root = bench.canonical_symmetry(p.k, p.edges)
    return sge.plan(p, stats, symmetry_seq=seq, root_edge=root, **kw)


@pytest.mark.parametrize("exploration", [False, True])
@pytest.mark.parametrize("iep", [False, True])
@pytest.mark.parametrize("scale,m,stride,cap", [(9, 4000, 11, 0), (11, 20000, 97, 300), (13, 90000, 4999, 0)])
def test_dense_roots_count_as_lists(sge, scale, m, stride, cap, iep, exploration):
    ks = [(5, 10), (5, 9), (5, 8)] + [(6, 9 + i % 6) for i in range(24)] + [(7, 14 + i % 6) for i in range(18)]
    if cap == 0 and scale > 11:
        ks = [(5, 10), (6, 13), (6, 14), (6, 12), (6, 15), (5, 9)]
    pats = [sge.PatternGraph.random(k, e, 700 + i) for i, (k, e) in enumerate(ks)]
    with sge.Engine(sge.gen_rmat(scale, m, seed=scale)) as eng:
        plans = [rooted(sge, p, eng, iep=iep, exploration=exploration) for p in pats]
        opts = dict(root_stride=stride, root_offset=3, root_max_degree=cap)
        got, inst, st = eng.count(plans, **opts)
        want, winst, _ = eng.count(plans, max_level_capacity=eng.info()["max_degree"], **opts)
        with eng.batch(plans, **opts) as b:
            again = [b.run()[0] for _ in range(2)]
    assert st["gpu_launches"] >= 5  # the bitset kernels ran
    assert got == want and inst == winst
    assert again == [want, want]
    assert sum(got) > 0


@pytest.mark.parametrize("k,m", [(5, 10), (6, 12), (6, 14), (7, 17), (7, 21), (8, 24)])
def test_dense_counts_match_the_oracle(sge, oracle, k, m):
    g = sge.gen_chung_lu(600, 3000, 2.1, 150, seed=5)
    plans = [sge.plan(sge.PatternGraph.random(k, m, s), g, iep=iep) for s in (1, 2) for iep in (False, True)]
    with sge.Engine(g) as eng:
        got, _, _ = eng.count(plans)
    want = [oracle.count_plan(g.offsets, g.nbrs, b, threads=0)[0] * b.count_multiplier % 2 ** 64 for b in plans]
    assert got == want


MIRROR_PATTERNS = {
    "triangle": (3, [(0, 1), (0, 2), (1, 2)]),
    "cycle4": (4, [(0, 1), (1, 2), (2, 3), (0, 3)]),
    "k4": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]),
    "star3": (4, [(0, 1), (0, 2), (0, 3)]),
    "house": (5, [(0, 1), (0, 2), (0, 4), (1, 3), (1, 4), (2, 3)]),
    "k5_minus_e": (5, [(a, b) for a in range(5) for b in range(a + 1, 5) if (a, b) != (3, 4)]),
    "bull": (5, [(0, 1), (0, 2), (1, 2), (1, 3), (2, 4)]),
}


@pytest.mark.parametrize("exploration", [False, True])
@pytest.mark.parametrize("reverse", [False, True])
def test_counts_do_not_depend_on_the_id_order(sge, oracle, reverse, exploration):
    """Hubs at low ids (the reversed restrictions run) and at high ids (the
    plan's own), with and without inclusion-exclusion."""
    g = sge.gen_rmat(9, 3000, seed=3)
    if reverse:
        g = sge.DataGraph.from_edges(g.num_vertices - 1 - g.edge_array().astype("int64"), g.num_vertices)
    plans = [sge.plan(sge.PatternGraph.from_edges(k, e), g, iep=iep, exploration=exploration)
             for k, e in MIRROR_PATTERNS.values() for iep in (False, True)]
    with sge.Engine(g) as eng:
        got, _, _ = eng.count(plans)
        split, _, _ = eng.count(plans, heavy_threshold=32)
    want = [oracle.count_plan(g.offsets, g.nbrs, b, threads=0)[0] * b.count_multiplier for b in plans]
    assert got == want and split == want


INLINE_PATTERNS = {
    "house": MIRROR_PATTERNS["house"],
    "cycle4_tail": (5, [(0, 1), (1, 2), (2, 3), (0, 3), (0, 4)]),
    "cycle4_far_tail": (5, [(0, 1), (1, 2), (2, 3), (0, 3), (2, 4)]),
    "cycle5": (5, [(0, 1), (1, 2), (2, 3), (3, 4), (0, 4)]),
    "path_triangle": (5, [(0, 1), (1, 2), (2, 3), (1, 3), (0, 4)]),
    "near5clique_8e": (5, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (1, 3), (1, 4), (2, 3)]),
}


@pytest.mark.parametrize("exploration", [False, True])
@pytest.mark.parametrize("n,m,maxd", [(300, 2500, 120), (3000, 9000, 900), (33_000, 40_000, 1500)])
def test_inline_tails(sge, oracle, n, m, maxd, exploration):
    """Tails that do not depend on the last enumerated level: by words of the
    hub bitmaps (small n), by a scan per candidate (no shared-memory tables
    beyond 32,768 vertices), hub and list candidates side by side."""
    g = sge.gen_chung_lu(n, m, 2.1, maxd, seed=n)
    plans = [sge.plan(sge.PatternGraph.from_edges(k, e), g, iep=iep, exploration=exploration)
             for k, e in INLINE_PATTERNS.values() for iep in (False, True)]
    opts = dict(root_stride=7, root_offset=2) if n > 300 else {}
    with sge.Engine(g) as eng:
        got, _, _ = eng.count(plans, **opts)
        split, _, _ = eng.count(plans, heavy_threshold=32, **opts)
        lists, _, _ = eng.count(plans, hub_bitmaps=False, **opts)
    raw = b"".join(b.to_bytes() for b in plans)
    want, _ = oracle.count_plans(g.offsets, g.nbrs, raw, len(plans), stride=opts.get("root_stride", 1),
                                 offset=opts.get("root_offset", 0))
    want = [w * b.count_multiplier for w, b in zip(want, plans)]
    assert got == want and split == want and lists == want
