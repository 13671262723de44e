"""Support group 0: vertices on both sides of the 16 in-edges and 16 row entries from which they get a table, on
graphs of any size, from a path to cliques; counts and decompositions as with lane groups and as the oracle's."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _layers(a, b, c):
    """Three layers, each vertex joined to all of the next ones: the middle one has a lower and c higher neighbours."""
    u, v = np.triu_indices(a + b + c, 1)
    layer = np.searchsorted([a, a + b], np.arange(a + b + c), side="right")
    keep = layer[u] != layer[v]
    return a + b + c, u[keep], v[keep]


def _union(*parts):
    us, vs, base = [], [], 0
    for n, u, v in parts:
        us.append(np.asarray(u, np.int64) + base)
        vs.append(np.asarray(v, np.int64) + base)
        base += n
    return base, np.concatenate(us).astype(np.uint32), np.concatenate(vs).astype(np.uint32)


GRAPHS = {
    "path": lambda: (70001, np.arange(70000, dtype=np.uint32), np.arange(1, 70001, dtype=np.uint32)),
    "layers": lambda: _union(*[_layers(a, b, c) for a in (15, 16, 17) for b in (40, 70) for c in (15, 16, 17)]),
    "cliques": lambda: _union(*[(s, *np.triu_indices(s, 1)) for s in (2, 16, 17, 31, 32, 33, 34, 60)]),
    "ws": lambda: kt.gen_ws(20000, 30, 0.2, 3),
    "rmat13": lambda: kt.gen_rmat(13, 16, 0.57, 0.19, 0.19, 11),
}


@pytest.mark.parametrize("name", GRAPHS)
def test_group_0(name):
    torch = pytest.importorskip("torch")
    n, u, v = GRAPHS[name]()
    src, dst = both_directions(u, v)
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    triangles = set()
    for limit in (None, 0):  # the list fill counts again
        eng.set_list_limit(limit)
        for group in (0, 8):
            eng.set_schedule(group, 32, 85, 50, 0)
            out.fill_(-1)
            torch.cuda.synchronize()
            eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, out.data_ptr())
            assert np.array_equal(out.cpu().numpy().view(np.uint32), ref["truss"]), (limit, group)
            triangles.add(eng.stats().triangles)
    assert len(triangles) == 1
    eng.close()
