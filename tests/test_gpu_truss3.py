"""The 3-truss in one pass over the supports: edge counts that are no multiple of four, graphs in which
all, none or some of the edges are in triangles, more edges than one sweep of the grid takes."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions, edge_keys

pytestmark = pytest.mark.gpu


def _graph(kind, edges):
    if kind == "path":  # no triangle
        i = np.arange(edges)
        return edges + 1, i, i + 1
    if kind == "fan":  # a hub, and a path through the other vertices: every edge but a last odd one in a triangle
        half = (edges + 1) // 2
        rim = np.arange(1, half + 1)
        u, v = np.concatenate([np.zeros(half, int), rim[:-1]]), np.concatenate([rim, rim[:-1] + 1])
        tail = edges - len(u)
        return half + 1 + tail, np.concatenate([u, np.full(tail, half)]), np.concatenate([v, half + 1 + np.arange(tail)])
    n, u, v = kt.gen_rmat(max(4, int(edges).bit_length() - 1), 8, 0.57, 0.19, 0.19, 3)
    return n, u[:edges], v[:edges]


@pytest.mark.parametrize("kind", ["path", "fan", "rmat"])
@pytest.mark.parametrize("edges", [1, 2, 3, 4, 5, 1023, 1024, 1025, 4097, 300_003, 1_300_001])
def test_truss3(edges, kind):
    torch = pytest.importorskip("torch")
    n, u, v = (np.asarray(x) for x in _graph(kind, edges))
    u, v = u.astype(np.uint32), v.astype(np.uint32)
    src, dst = both_directions(u, v)
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda() for a in (src, dst))
    d_keep = torch.full((len(src),), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for orientation in ("directed-by-degree", "directed-by-index"):
        eng.set_variant(directedness=orientation)
        for run in (lambda: eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), int(n), 3, d_keep.data_ptr()),
                    eng.replay):
            d_keep.fill_(7)
            torch.cuda.synchronize()
            run()
            keep = d_keep.cpu().numpy()
            want = edge_keys(*oracle.ktruss(int(n), src, dst, 3))
            assert np.array_equal(edge_keys(src[keep == 1], dst[keep == 1]), want) and keep.max() <= 1
            gone = len(u) - len(want)
            st, log = eng.stats(), eng.round_log()
            assert (st.num_rounds, st.num_levels) == (int(gone > 0), 1) and list(log["size"]) == [gone] * (gone > 0)
    eng.close()
