"""The tuple sort's key widths (64-bit keys, 128-bit keys, rows wider than both)
and tile edges, tries of several levels across tiles, and device ingest of
edge lists with repeats and self-loops, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()


# bits per column: 63/64/65 and 127/128/129 bits in all, columns that are all zero, one bit, 32 bits
WIDTHS = [(32, 31), (32, 32), (32, 32, 1), (13,) * 5, (0, 7, 0), (1,), (32,) * 4, (32, 32, 32, 31), (32,) * 4 + (1,),
          (20, 32, 9, 0, 32, 32, 17)]


@pytest.mark.parametrize("n", [2, 255, 2048, 2049, 4096, 4097, 40_003])
@pytest.mark.parametrize("widths", WIDTHS)
def test_sort_key_widths_and_tile_edges(sge, widths, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + len(widths))
    a = np.stack([rng.integers(0, 1 << w, size=n, dtype=np.uint64).astype(np.uint32) for w in widths], 1)
    a[rng.integers(0, n, size=n // 3)] = a[0]                      # repeated rows
    for c, w in enumerate(widths):
        a[-1, c] = (1 << w) - 1                                   # every column's width is in use
    d = _dev(torch, a)
    sge.sort_tuples_device(d.data_ptr(), n, len(widths))
    got = d.cpu().numpy().view(np.uint32).reshape(n, len(widths))
    assert np.array_equal(got, a[np.lexsort(a.T[::-1])])


@pytest.mark.parametrize("n,arity,hi", [(1, 1, 5), (1023, 2, 40), (1025, 4, 6), (30_000, 3, 50), (30_000, 6, 4)])
def test_trie_levels_across_tiles(sge, n, arity, hi):
    torch = pytest.importorskip("torch")
    rows = np.random.default_rng(n).integers(0, hi, size=(n, arity)).astype(np.uint32)
    rows = rows[np.lexsort(rows.T[::-1])]                         # (repeated rows stay)
    d = _dev(torch, rows)
    t = sge.trie_build_device(d.data_ptr(), n, arity)
    try:
        starts = []
        for lvl in range(arity):
            new = np.ones(n, bool)
            new[1:] = np.any(rows[1:, : lvl + 1] != rows[:-1, : lvl + 1], axis=1)
            starts.append(np.nonzero(new)[0])
        for lvl in range(arity):
            vals, child = sge.trie_level(t, lvl)
            assert np.array_equal(vals, rows[starts[lvl], lvl])
            if lvl + 1 < arity:
                want = np.searchsorted(starts[lvl + 1], np.append(starts[lvl], n))
                assert np.array_equal(child.astype(np.int64), want)
    finally:
        sge.trie_free(t)


@pytest.mark.parametrize("n,m", [(2, 5), (3, 40), (1 << 10, 2048), (1000, 2049), ((1 << 16) + 1, 100_003)])
def test_ingest_drops_repeats_and_self_loops(sge, n, m):
    torch = pytest.importorskip("torch")
    e = np.random.default_rng(m).integers(0, n, size=(m, 2)).astype(np.uint32)
    e[: m // 4] = e[m // 4: 2 * (m // 4)][:, ::-1]                # reversed repeats
    e[-1] = n - 1                                                # a self-loop of the last id
    d = _dev(torch, e)
    want = sge.DataGraph.from_edges(e, n)
    with sge.Engine.from_device_edges(d.data_ptr(), m, n) as eng:
        off, nb = eng.csr()
    assert np.array_equal(off, want.offsets) and np.array_equal(nb, want.nbrs)


@pytest.mark.parametrize("kind", ["rmat", "chung_lu", "star", "path", "isolated"])
def test_graph_handle_facts_match_the_host(sge, kind):
    """Root edges (through counts), planner statistics and hub index of a
    device graph, against the host's own: degree moments and wedge sample give
    the same plan costs bit for bit."""
    g = {"rmat": lambda: sge.gen_rmat(12, 30_001, seed=2), "chung_lu": lambda: sge.gen_chung_lu(5000, 30_000, 2.1, 0, 4),
         "star": lambda: sge.DataGraph.from_edges(np.array([(0, i) for i in range(1, 3000)]), 3000),
         "path": lambda: sge.DataGraph.from_edges(np.array([(i, i + 1) for i in range(2047)]), 2048),
         "isolated": lambda: sge.DataGraph.from_edges(np.array([(5, 900), (5, 1023), (900, 1023)]), 4100)}[kind]()
    pats = [sge.PatternGraph.random(k, m, 40 + k) for k, m in ((3, 3), (4, 4), (5, 7), (6, 11), (7, 16))]
    stats = g.stats()
    with sge.Engine(g) as eng:
        info = eng.info()
        for p in pats:
            a, b = sge.plan(p, eng), sge.plan(p, stats)
            assert a.to_bytes() == b.to_bytes()
        deg = np.diff(g.offsets)
        if info["hub_count"]:
            assert info["hub_count"] == int((deg >= info["hub_min_degree"]).sum())
        hubs, _, _ = eng.count([sge.plan(pats[0], eng)])
        lists, _, _ = eng.count([sge.plan(pats[0], eng)], hub_bitmaps=False)
    assert hubs == lists
    if kind == "isolated":
        assert hubs == [6]
