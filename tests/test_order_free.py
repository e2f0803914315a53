"""Which plans may be counted with all bounds reversed (sge_plan_order_free):
checked against the definition, every order of a small pattern's ids."""
import itertools
import random

import pytest


def adjacency(b):
    k = b.k
    adj = [[False] * k for _ in range(k)]
    for i in range(1, k):
        for j in range(i):
            if (b.parents[i] >> j) & 1:
                adj[i][j] = adj[j][i] = True
    return adj


def kept_per_order(b, labels=None):
    """Over every order of k ids: how many automorphic images satisfy the bounds."""
    k = b.k
    adj = adjacency(b)
    lab = [0] * k if labels is None else [labels[b.order[i]] for i in range(k)]
    auts = [s for s in itertools.permutations(range(k))
            if all(adj[s[i]][s[j]] == adj[i][j] for i in range(k) for j in range(i))
            and all(lab[s[i]] == lab[i] for i in range(k))]
    pairs = []
    if b.root_kind == 1:
        pairs.append((0, 1))
    if b.root_kind == 2:
        pairs.append((1, 0))
    for i in range(2, k):
        for j in range(k):
            if (b.lower[i] >> j) & 1:
                pairs.append((j, i))
            if (b.upper[i] >> j) & 1:
                pairs.append((i, j))
    return {sum(all(o[s[x]] < o[s[y]] for x, y in pairs) for s in auts) for o in itertools.permutations(range(k))}


def random_pattern(sge, rng, k):
    m = rng.randint(k - 1, k * (k - 1) // 2)
    return sge.PatternGraph.random(k, m, rng.randrange(1 << 20))


@pytest.mark.parametrize("k", [3, 4, 5, 6, 7, 8])
def test_every_planned_blob_is_order_free(sge, k):
    rng = random.Random(k)
    for _ in range(12 if k < 8 else 4):
        p = random_pattern(sge, rng, k)
        for iep in (False, True):
            for b in sge.candidates(p, None, iep=iep, cap=64):
                assert sge.plan_order_free(b)
    labels = [rng.randrange(2) for _ in range(k)]
    p = random_pattern(sge, rng, k)
    assert all(sge.plan_order_free(b, labels) for b in sge.candidates(p, None, labels=labels))


@pytest.mark.parametrize("k", [9, 12, 16])
def test_large_patterns(sge, k):
    star = sge.PatternGraph.from_edges(k, [(0, i) for i in range(1, min(k, 9))] + [(i, i + 1) for i in range(8, k - 1)])
    cycle = sge.PatternGraph.from_edges(k, [(i, (i + 1) % k) for i in range(k)])
    for p in (star, cycle):
        assert all(sge.plan_order_free(b) for b in sge.candidates(p, None, cap=8))


@pytest.mark.parametrize("k", [3, 4, 5])
def test_edited_bounds_against_the_definition(sge, k):
    """Bounds dropped, added and reversed: a plan called order free keeps as
    many images under every order of the ids."""
    rng = random.Random(100 + k)
    free = bound = 0
    for _ in range(150):
        b = sge.PlanBlob.from_bytes(sge.plan(random_pattern(sge, rng, k), None, iep=False).to_bytes())
        for i in range(2, k):
            for j in range(i):
                lo, up, bit = b.lower[i], b.upper[i], 1 << j
                pick = rng.choice(["keep", "drop", "lower", "upper"])
                if pick == "drop":
                    lo, up = lo & ~bit, up & ~bit
                elif pick == "lower":
                    lo, up = lo | bit, up & ~bit
                elif pick == "upper":
                    lo, up = lo & ~bit, up | bit
                b.lower[i], b.upper[i] = lo, up
            b.check[i] = ((1 << i) - 1) & ~(b.parents[i] | b.lower[i] | b.upper[i])
        b.root_kind = rng.choice([0, b.root_kind])
        if b.root_kind == 0:
            b.lower[1] = b.upper[1] = 0
        sge.validate_plan(b)
        kept = kept_per_order(b)
        if sge.plan_order_free(b):
            free += 1
            assert len(kept) == 1
        bound += len(kept) > 1
    assert free >= 10 and bound >= 10


def test_wedge_below_one_leaf_only(sge):
    b = sge.plan(sge.PatternGraph.from_edges(3, [(0, 1), (0, 2)]), None, iep=False, force_order=[0, 1, 2])
    for i in (1, 2):
        b.lower[i] = b.upper[i] = 0
    b.check[2] = 2
    assert sge.plan_order_free(b)   # no bounds: every embedding
    b.root_kind, b.lower[1] = 1, 1
    assert not sge.plan_order_free(b)


def test_other_tail_sums_and_labels(sge):
    """Inclusion-exclusion with other coefficients counts something else; a
    labeled plan is judged by the labels it gets."""
    star = sge.PatternGraph.from_edges(5, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 4)])
    iep = [b for b in sge.candidates(star, None, cap=64) if b.tail_mode == 3]
    assert iep
    b = sge.PlanBlob.from_bytes(iep[0].to_bytes())
    b.part_coef[1] = 0
    assert not sge.plan_order_free(b)
    tri = sge.PatternGraph.from_edges(3, [(0, 1), (0, 2), (1, 2)])
    b = sge.plan(tri, None, labels=[4, 4, 4])
    assert sge.plan_order_free(b, [4, 4, 4])
    assert not sge.plan_order_free(b, [4, 4, 5])
    with pytest.raises(sge.SgeError):
        sge.plan_order_free(b)
