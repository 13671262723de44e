"""The vertex-centric support count and list fill where their batches of 256 in-edges, their warps'
shares and their rows' tables end: vertices with that many in-edges and rows, tails of all lengths."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions, edge_keys

pytestmark = pytest.mark.gpu


def _graph(core, pages, tails, seed):
    """A clique of `core` vertices of the highest degrees, each with in-edges from `pages` vertices whose
    tails hold up to `tails` core vertices (some none: pages with one edge), and a few edges between
    pages."""
    rng = np.random.default_rng(seed)
    cu, cv = np.triu_indices(core, 1)
    us, vs = [cu], [cv]
    for p in range(pages):
        k = int(rng.integers(1, min(tails, core) + 1))
        # consecutive core vertices from anywhere: every in-edge's tail ends at another place
        first = int(rng.integers(0, core - k + 1))
        us.append(np.arange(first, first + k))
        vs.append(np.full(k, core + p))
    extra = rng.integers(0, pages, (2, pages // 4))
    extra = extra[:, extra[0] != extra[1]] + core
    us.append(extra.min(0))
    vs.append(extra.max(0))
    keys = np.unique(np.concatenate(us).astype(np.uint64) << np.uint64(32) | np.concatenate(vs).astype(np.uint64))
    return core + pages, (keys >> np.uint64(32)).astype(np.uint32), (keys & np.uint64(0xffffffff)).astype(np.uint32)


@pytest.mark.parametrize("core,tails", [(1, 1), (2, 2), (33, 33), (128, 5), (300, 300)])
@pytest.mark.parametrize("pages", [1, 255, 256, 257, 513])
def test_batches(pages, core, tails):
    torch = pytest.importorskip("torch")
    n, u, v = _graph(core, pages, tails, [pages, core])
    src, dst = both_directions(u, v)
    eng = kt.Engine(0)
    eng.set_schedule(support_group=0)  # every vertex is counted that way, in a graph of any size
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda() for a in (src, dst))
    d_truss = torch.zeros(len(src), dtype=torch.int32, device="cuda")
    d_keep = torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_truss.data_ptr())
    assert np.array_equal(d_truss.cpu().numpy().view(np.uint32), oracle.decompose(n, src, dst, method="peel")["truss"])
    for k in (3, 4, 12):
        eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, d_keep.data_ptr())
        keep = d_keep.cpu().numpy().astype(bool)
        assert np.array_equal(edge_keys(src[keep], dst[keep]), edge_keys(*oracle.ktruss(n, src, dst, k)))
    eng.close()
