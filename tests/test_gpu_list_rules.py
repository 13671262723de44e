"""Which decompositions peel from lists and which walk: near-cliques on both sides of the rule, alone and
beside other graphs, and densities on both sides of its line.  Either way the truss numbers are the
oracle's, and a replay takes the same way."""
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


def _rewired(graph, share):
    n, u, v = graph
    rng = np.random.default_rng(1)
    u, v = u.astype(np.int64), v.astype(np.int64)
    moved = rng.random(len(u)) < share
    v[moved] = rng.integers(0, n, moved.sum())
    keys = np.unique(np.minimum(u, v) * n + np.maximum(u, v))
    keys = keys[keys // n != keys % n]
    return n, keys // n, keys % n


def _beside(*parts):
    base, us, vs = 0, [], []
    for n, u, v in parts:
        us.append(np.asarray(u, np.int64) + base)
        vs.append(np.asarray(v, np.int64) + base)
        base += n
    return base, np.concatenate(us), np.concatenate(vs)


@pytest.mark.parametrize("name,graph,lists", [
    ("cliques of 60", lambda: _cliques(60, 160), False),
    ("cliques of 20: few entries", lambda: _cliques(20, 1500), True),
    ("cliques of 60, a tenth rewired", lambda: _rewired(_cliques(60, 160), 0.1), True),
    ("mostly cliques", lambda: _beside(_cliques(200, 16), kt.gen_rmat(11, 8, 0.57, 0.19, 0.19, 2)), False),
    ("half cliques", lambda: _beside(_cliques(60, 80), kt.gen_rmat(14, 16, 0.57, 0.19, 0.19, 2)), True),
    ("few edges in cliques", lambda: _cliques(60, 140), True),
    ("dense", lambda: kt.gen_er(900, 0.75, 3), True),
    ("denser", lambda: kt.gen_er(900, 0.85, 3), False),
])
def test_rules(name, graph, lists):
    torch = pytest.importorskip("torch")
    n, u, v = (np.asarray(x) for x in graph())
    n, u, v = int(n), u.astype(np.uint32), v.astype(np.uint32)
    assert len(u) > 1 << 17
    src, dst = both_directions(u, v)
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).cuda() for x in (src, dst))
    d_out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    want = oracle.decompose(n, src, dst, method="peel")["truss"]
    for run in (lambda: eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_out.data_ptr()),
                eng.replay, eng.replay):
        d_out.fill_(-1)
        torch.cuda.synchronize()
        run()
        assert np.array_equal(d_out.cpu().numpy().view(np.uint32), want), name
    # every edge's list is queued once; a walk queues rows, which are longer
    st = eng.stats()
    assert (st.walk_entries == 3 * st.triangles) == lists
    eng.close()
