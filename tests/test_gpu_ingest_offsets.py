"""Device edge lists that start at any 32-bit word of a larger buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 5000])
@pytest.mark.parametrize("words", [1, 2, 3])
def test_device_edges_behind_a_header(sge, words, m):
    torch = pytest.importorskip("torch")
    n = 300
    e = np.random.default_rng(words).integers(0, n, size=(m, 2), dtype=np.uint32)
    d = torch.from_numpy(np.concatenate([np.full(words, n + 7, np.uint32), e.ravel()]).view(np.int32)).cuda()
    with sge.Engine.from_device_edges(d.data_ptr() + 4 * words, m, n) as eng:
        off, nb = eng.csr()
    host = sge.DataGraph.from_edges(e, n, dedup=True)
    assert np.array_equal(off, host.offsets)
    assert np.array_equal(nb, host.nbrs)
