"""Graphs of fewer than 2^18 edges on both sides of the rules that send them to the walks: near-cliques by
their list entries and by what lies beside them, others by their density and evenness.  The truss numbers
are the oracle's, a replay goes the same way."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _cliques(size, count):
    u, v = np.triu_indices(size, 1)
    at = size * np.arange(count)[:, None]
    return size * count, (u + at).ravel(), (v + at).ravel()


def _beside(*parts):
    base, us, vs = 0, [], []
    for n, u, v in parts:
        us.append(np.asarray(u, np.int64) + base)
        vs.append(np.asarray(v, np.int64) + base)
        base += n
    return base, np.concatenate(us), np.concatenate(vs)


def _rmat(scale, ef):
    return kt.gen_rmat(scale, ef, 0.57, 0.19, 0.19, 2)


@pytest.mark.parametrize("name,graph,lists", [
    ("many entries", lambda: _cliques(400, 2), False),
    ("the most", lambda: _cliques(500, 2), False),
    ("past the line", lambda: _cliques(200, 6), False),
    ("below the line", lambda: _cliques(100, 26), True),
    ("beside few triangles", lambda: _beside(_cliques(500, 2), _rmat(10, 4)), False),
    ("beside many", lambda: _beside(_cliques(200, 5), _rmat(12, 8)), True),
    ("dense", lambda: kt.gen_er(700, 0.64, 3), True),       # 287 entries an edge
    ("denser", lambda: kt.gen_er(700, 0.72, 3), False),     # 363
    ("denser, uneven", lambda: kt.gen_ba(700, 350, 3), True),   # about 400, but of 200 to 500 by edge
    ("beside a sparse graph", lambda: _beside(_cliques(300, 2), kt.gen_er(20000, 4e-4, 3)), False),
])
def test_small_near_cliques(name, graph, lists):
    torch = pytest.importorskip("torch")
    n, u, v = graph()
    n, u, v = int(n), u.astype(np.uint32), v.astype(np.uint32)
    assert 1 << 15 < len(u) < 1 << 18
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
