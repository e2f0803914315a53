"""Degree statistics of a graph with one vertex of huge degree: the same sums,
in vertex order, in memory that does not grow with that degree."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

CODE = """
import resource, sys
sys.path.insert(0, sys.argv[1])
import ctypes as C
import numpy as np
import sge
n, d = 1 << 22, (1 << 21) - 1          # vertex 0 meets 1..d, the others none
off = np.minimum(np.arange(n + 1, dtype=np.int64) - 1 + d, 2 * d).astype(np.uint32)
off[0] = 0
nb = np.zeros(2 * d, np.uint32)
nb[:d] = np.arange(1, d + 1)
st = sge.GraphStats()
sge.lib().sge_graph_stats_compute(sge._u32p(off[:3].copy() * 0), sge._u32p(nb), 2, C.byref(st))
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
assert sge.lib().sge_graph_stats_compute(sge._u32p(off), sge._u32p(nb), n, C.byref(st)) == 0
print(resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before, st.max_degree, st.moments[0], st.moments[1])
"""


def test_one_huge_degree(sge):
    pkg = Path(sge.__file__).resolve().parent
    r = subprocess.run([sys.executable, "-c", CODE, str(pkg)], capture_output=True, text=True, check=True)
    grown_kb, maxd, m0, m1 = map(float, r.stdout.split())
    d = (1 << 21) - 1
    assert (maxd, m0, m1) == (d, 1 << 22, 2 * d)
    # the wedge sample's prefix sums (8 bytes a vertex) and a small table, not 18 doubles a degree (302 MB)
    assert grown_kb < 100_000


@pytest.mark.parametrize("n,hub", [(10, 9), (9000, 4095), (9000, 4096), (9000, 4400), (9000, 8000)])
def test_moments_are_the_plain_sums(sge, n, hub):
    rng = np.random.default_rng(n + hub)
    e = rng.integers(0, n, size=(3 * n, 2))
    e = np.concatenate([e, np.stack([np.zeros(hub, np.int64), np.arange(1, hub + 1)], 1)])
    g = sge.DataGraph.from_edges(e.astype(np.uint32), n, dedup=True)
    st = g.stats()
    want = np.zeros(len(st.moments))
    for d in np.diff(g.offsets.astype(np.int64)):
        p = 1.0
        for j in range(want.size):
            want[j] += p
            p *= float(d)
    assert list(st.moments) == list(want)
