"""Graphs whose triangles lie in a dense part, beside edges in none: even parts walk, uneven and thinner ones take
lists.  The truss numbers are the oracle's, a replay goes the same way."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _tree(m):
    return m + 1, np.arange(1, m + 1) // 4, np.arange(1, m + 1)


def _clique(size):
    u, v = np.triu_indices(size, 1)
    return size, u, v


def _beside(*parts):
    base, us, vs = 0, [], []
    for n, u, v in parts:
        us.append(np.asarray(u, np.int64) + base)
        vs.append(np.asarray(v, np.int64) + base)
        base += n
    return base, np.concatenate(us), np.concatenate(vs)


def _core(left, right, clique):
    """A complete bipartite graph with a clique on its left side."""
    a, b = np.divmod(np.arange(left * right), right)
    i, j = np.triu_indices(clique, 1)
    return left + right, np.concatenate([a, i]), np.concatenate([b + left, j])


@pytest.mark.parametrize("name,graph,lists", [
    ("core", lambda: _core(2000, 900, 450), False),          # 630 entries an edge in triangles, 0.71 of the mean
    ("small core", lambda: _core(1500, 600, 200), True),
    ("clique", lambda: _beside(_tree(900000), _clique(540)), False),
    # 478 entries an edge in triangles, but 54 an edge of the whole graph, all of them of a near-clique
    ("smaller clique", lambda: _beside(_tree(900000), _clique(480)), False),
    ("even", lambda: _beside(_tree(900000), kt.gen_er(1000, 0.75, 3)), False),
    ("uneven", lambda: _beside(_tree(900000), kt.gen_ba(1500, 600, 3)), True),
])
def test_dense_parts(name, graph, lists):
    torch = pytest.importorskip("torch")
    n, u, v = graph()
    n, u, v = int(n), u.astype(np.uint32), v.astype(np.uint32)
    assert len(u) > 1 << 18
    src, dst = both_directions(u, v)
    want = oracle.decompose(n, src, dst, method="peel")["truss"]
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).cuda() for x in (src, dst))
    out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    for run in (lambda: eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, out.data_ptr()),
                eng.replay, eng.replay):
        out.fill_(-1)
        torch.cuda.synchronize()
        run()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        st = eng.stats()
        assert (st.walk_entries == 3 * st.triangles) == lists
    eng.close()
