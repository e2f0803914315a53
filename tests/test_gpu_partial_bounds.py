"""Plans whose bounds are not a full symmetry breaking (sge_plan_create takes
any consistent masks): the count is defined by the id order, so a full run, its
shards, the instrumented run, a capped run and the oracle agree on it, on
graphs with the hubs at low and at high ids."""
import itertools

import pytest

pytestmark = pytest.mark.gpu


def edited(sge, k, edges, bounds, order):
    """The pattern's plan in `order` with only these (small, large) level pairs as bounds."""
    b = sge.PlanBlob.from_bytes(sge.plan(sge.PatternGraph.from_edges(k, edges), None, iep=False,
                                         force_order=order).to_bytes())
    b.count_multiplier = 1
    b.root_kind = 0
    for i in range(1, k):
        b.lower[i] = b.upper[i] = 0
    for s, l in bounds:
        if s < l:
            b.lower[l] |= 1 << s
        else:
            b.upper[s] |= 1 << l
    b.root_kind = 1 if b.lower[1] else 2 if b.upper[1] else 0
    for i in range(1, k):
        b.check[i] = ((1 << i) - 1) & ~(b.parents[i] | b.lower[i] | b.upper[i])
    sge.validate_plan(b)
    return b


def plans(sge):
    k4 = list(itertools.combinations(range(4), 2))
    k5 = list(itertools.combinations(range(5), 2))
    return [
        edited(sge, 3, [(0, 1), (0, 2)], [(0, 1)], [0, 1, 2]),                # a wedge, centre below one leaf
        edited(sge, 3, [(0, 1), (0, 2), (1, 2)], [(0, 1), (0, 2)], [0, 1, 2]),  # its lowest vertex first: complete in part
        edited(sge, 4, [(0, 1), (1, 2), (2, 3)], [(0, 1), (1, 2)], [1, 0, 2, 3]),
        edited(sge, 4, [(0, 1), (1, 2), (2, 3), (0, 3)], [(0, 1), (0, 2)], [0, 1, 2, 3]),
        edited(sge, 4, k4, [(0, 1)], [0, 1, 2, 3]),
        edited(sge, 5, k5, [(0, 1), (1, 3)], [0, 1, 2, 3, 4]),
        edited(sge, 5, [(0, 1), (0, 2), (0, 4), (1, 3), (1, 4), (2, 3)], [(0, 1), (0, 3)], [0, 1, 2, 3, 4]),
    ]


@pytest.mark.parametrize("reverse", [False, True])
def test_partial_bounds_keep_their_direction(sge, oracle, reverse):
    g = sge.gen_rmat(9, 3000, seed=3)
    if reverse:
        g = sge.DataGraph.from_edges(g.num_vertices - 1 - g.edge_array().astype("int64"), g.num_vertices)
    ps = plans(sge)
    want = [oracle.count_plan(g.offsets, g.nbrs, b, threads=0)[0] for b in ps]
    with sge.Engine(g) as eng:
        full, _, _ = eng.count(ps)
        shards = [eng.count(ps, root_stride=3, root_offset=i)[0] for i in range(3)]
        counted, _, _ = eng.count(ps, stats=True)
        capped, _, _ = eng.count(ps, max_level_capacity=eng.info()["max_degree"])
        with eng.batch(ps) as b:
            batch = b.run()[0]
    assert [sum(s) for s in zip(*shards)] == want
    assert counted == want and capped == want
    assert full == want and batch == want


def test_contradictory_bounds_count_nothing(sge, oracle):
    """Above and below the same vertex: sge_plan_validate takes it, no vertex fits."""
    g = sge.gen_rmat(9, 3000, seed=3)
    out = []
    for k, edges in ((5, list(itertools.combinations(range(5), 2))), (6, list(itertools.combinations(range(6), 2)))):
        for lv in (2, 3, k - 1):
            b = edited(sge, k, edges, [], list(range(k)))
            b.lower[lv] |= 2
            b.upper[lv] |= 2
            sge.validate_plan(b)
            out.append(b)
    want = [oracle.count_plan(g.offsets, g.nbrs, b, threads=0)[0] for b in out]
    assert want == [0] * len(out)
    with sge.Engine(g) as eng:
        lists, _, _ = eng.count(out, max_level_capacity=eng.info()["max_degree"])
        full, _, _ = eng.count(out)
    assert lists == want and full == want
