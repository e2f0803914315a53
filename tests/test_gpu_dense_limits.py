"""Bit rows (csrc/dense.cuh) where a launch holds more root edges than it has
records for (2^17) or rows for (1 GB), and universes of more than 32 words.
Ring lattices, vertex i next to i ± 1 .. i ± w: every root edge has ends of
degree 2w >= 64, so every one is taken until a limit is met, and K5 has the
closed form n C(w, 4)."""
import itertools
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K5 = (5, list(itertools.combinations(range(5), 2)))
WHEEL4 = (5, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (2, 3), (3, 4), (1, 4)])
MAX_RECORDS, MAX_ROWS = 1 << 17, 1 << 30


def ring(sge, n, w):
    i = np.repeat(np.arange(n), w)
    return sge.DataGraph.from_edges(np.stack([i, (i + np.tile(np.arange(1, w + 1), n)) % n], 1), n)


def rows_bytes(words):
    return 16 * (1 + 16 * words + 32 * words * ((words + 3) // 4))


def test_more_roots_than_records(sge):
    n, w = 6000, 40
    assert n * w > MAX_RECORDS
    with sge.Engine(ring(sge, n, w)) as eng:
        for exploration in (False, True):
            b = sge.plan(sge.PatternGraph.from_edges(*K5), eng, iep=False, exploration=exploration)
            assert b.num_enum >= 4
            for _ in range(2):   # which roots get a record differs from run to run
                assert eng.count([b])[1][0] == n * math.comb(w, 4)


def test_more_rows_than_room(sge):
    n, w, stride = 3000, 200, 8
    # a root's common neighbours: 2w - 1 - distance, at least w - 1
    need = sum(rows_bytes(-(-(2 * w - 1 - d) // 32)) for d in range(1, w + 1)) * n // stride
    assert need > MAX_ROWS and n * w // stride < MAX_RECORDS
    with sge.Engine(ring(sge, n, w)) as eng:
        b = sge.plan(sge.PatternGraph.from_edges(*K5), eng, iep=False)
        got = eng.count([b], root_stride=stride)[1]
        want = eng.count([b], root_stride=stride, max_level_capacity=2 * w)[1]
        assert got == want and got[0] > 0


@pytest.mark.parametrize("exploration", [False, True])
def test_universes_of_two_words_a_lane(sge, exploration):
    n, w, stride = 3000, 560, 80021
    # N(u) holds 2w vertices, N(u) ∪ N(v) 4w less the common ones
    assert 1024 < 2 * w and 4 * w - (w - 1) + 96 <= 2048
    with sge.Engine(ring(sge, n, w)) as eng:
        b = sge.plan(sge.PatternGraph.from_edges(*WHEEL4), eng, iep=False, exploration=exploration)
        got = eng.count([b], root_stride=stride)[1]
        want = eng.count([b], root_stride=stride, max_level_capacity=2 * w)[1]
        assert got == want and got[0] > 0
