"""Replays and the buffer of the triangle lists: a graph of the same size with more triangles than the
buffer holds, put into the buffers of the call that is repeated, is refused and writes nothing."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def test_a_replay_whose_lists_outgrew_their_buffer():
    torch = pytest.importorskip("torch")
    n, size = 20000, 347  # a clique of 60,031 edges has 20.7 M list entries, the buffer 8.4 M
    u, v = (x.astype(np.uint32) for x in np.triu_indices(size, 1))
    m = len(u)
    clique = both_directions(u, v)
    rng = np.random.default_rng(5)
    keys = np.unique(rng.integers(0, n, 2 * m) * n + rng.integers(0, n, 2 * m))
    a, b = keys // n, keys % n
    keep = np.flatnonzero(a < b)
    keep = np.sort(rng.permutation(keep)[:m])
    sparse = both_directions(a[keep], b[keep])
    assert len(sparse[0]) == 2 * m
    want = oracle.decompose(n, *sparse, method="peel")["truss"]
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in sparse)
    truss = torch.full((2 * m,), -1, dtype=torch.int32, device="cuda")

    def put(graph):
        for d, x in zip((d_src, d_dst), graph):
            d.copy_(torch.from_numpy(x.view(np.int32)))
        truss.fill_(-1)
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), 2 * m, n, truss.data_ptr())
    assert eng.stats().walk_entries == 3 * eng.stats().triangles  # from lists
    for _ in range(2):
        put(clique)
        with pytest.raises(kt.KtrussError) as ei:
            eng.replay()
        assert ei.value.status == 1  # KT_ERR_INVALID_ARG
        assert bool((truss == -1).all())
    put(sparse)
    eng.replay()
    assert np.array_equal(truss.cpu().numpy().view(np.uint32), want)
    put(clique)
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), 2 * m, n, truss.data_ptr())
    assert bool((truss == size).all())
    eng.close()
