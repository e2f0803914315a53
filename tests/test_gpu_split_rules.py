"""The automatic choices of a counting launch against the plainer ones that the
options ask for, where those are the better: a launch that splits roots must
not take far longer than one that splits none, nor bit rows far longer than
lists.  Kernel times of the same process, best of several runs."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = {
    "tailed_triangle": (4, [(0, 1), (0, 2), (1, 2), (2, 3)]),
    "near5clique_8e": (5, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (1, 3), (1, 4), (2, 3)]),
    "wheel4": (5, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (2, 3), (3, 4), (1, 4)]),
    "k5": (5, list(itertools.combinations(range(5), 2))),
    "octahedron": (6, [e for e in itertools.combinations(range(6), 2) if e not in ((0, 1), (2, 3), (4, 5))]),
}
NO_SPLIT = 1 << 30


@pytest.fixture(scope="module")
def engines(sge):
    made = {}

    def get(name):
        if name not in made:
            if name == "sparse":     # mean degree 7, hubs of a few hundred
                g = sge.gen_chung_lu(300_000, 1_000_000, 2.3, 500, seed=6)
            elif name == "uniform":  # degree 200, 2 shared neighbours per edge
                e = np.random.default_rng(8).integers(0, 20_000, (2_000_000, 2))
                g = sge.DataGraph.from_edges(e, 20_000)
            else:
                g = sge.gen_rmat(16, 700_001, seed=2)
            made[name] = sge.Engine(g)
        return made[name]
    yield get
    for eng in made.values():
        eng.close()


def best(eng, b, **kw):
    ms, counts = [], set()
    for _ in range(6):
        c, _, st = eng.count([b], **kw)
        ms.append(st["kernel_ms"])
        counts.add(c[0])
    assert len(counts) == 1
    return min(ms[1:]), counts.pop()


def compare(sge, eng, name, limit, other, exploration=False, labels=None, **kw):
    k, edges = PATTERNS[name]
    pl = None if labels is None else [i % labels for i in range(k)]
    b = sge.plan(sge.PatternGraph.from_edges(k, edges), eng, iep=False, exploration=exploration, labels=pl)
    if pl is not None:
        kw["labels"] = [pl]
    auto, count = best(eng, b, **kw)
    plain, want = best(eng, b, **kw, **other)
    assert count == want
    assert auto <= limit * plain, f"{name}: {auto:.3f} ms, {plain:.3f} ms with {other}"


# a tail that is a range per candidate: 1.3 to 1.6 times longer when split
@pytest.mark.parametrize("exploration", [False, True])
def test_tail_in_one_list_is_not_split(sge, engines, exploration):
    compare(sge, engines("rmat"), "tailed_triangle", 1.15, dict(heavy_threshold=NO_SPLIT), exploration)


# weighed by degrees, these took 4 and 4 to 6 times as long
@pytest.mark.parametrize("exploration", [False, True])
@pytest.mark.parametrize("name", ["near5clique_8e", "wheel4"])
def test_roots_weigh_what_their_list_holds(sge, engines, name, exploration):
    lists = dict(max_level_capacity=engines("sparse").info()["max_degree"])
    compare(sge, engines("sparse"), name, 2.0, dict(heavy_threshold=NO_SPLIT), exploration, **lists)


# one root in 256 taken to carry the labels: 10 to 100 times as long
@pytest.mark.parametrize("labels", [2, 8, 32])
@pytest.mark.parametrize("graph", ["sparse", "uniform", "rmat"])
def test_labeled_roots_are_split_by_their_share(sge, engines, graph, labels):
    eng = engines(graph)
    eng.set_labels(np.random.default_rng(3).integers(0, labels, eng.info()["num_vertices"]))
    for name in ("k5", "wheel4", "octahedron") if graph != "rmat" else ("k5",):
        compare(sge, eng, name, 2.5, dict(heavy_threshold=NO_SPLIT), labels=labels)


# rows for every root: 1.3 to 8 times as long
@pytest.mark.parametrize("exploration", [False, True])
@pytest.mark.parametrize("graph,name,limit", [("sparse", "octahedron", 2.0), ("sparse", "wheel4", 2.0),
                                              ("sparse", "k5", 1.4), ("uniform", "octahedron", 1.3),
                                              ("uniform", "k5", 1.2)])
def test_rows_only_where_edges_share_neighbours(sge, engines, graph, name, limit, exploration):
    eng = engines(graph)
    compare(sge, eng, name, limit, dict(max_level_capacity=eng.info()["max_degree"]), exploration)
