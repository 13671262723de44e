"""Complete bipartite graphs with a clique on one side: tails of up to thousands over rows of the clique's size, on
both sides of the line that leaves them to the lane groups, in the count and in the three kernels of the list
fill."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _core(left, right, clique):
    a, b = np.divmod(np.arange(left * right), right)
    i, j = np.triu_indices(clique, 1)
    return left + right, np.concatenate([a, i]).astype(np.uint32), np.concatenate([b + left, j]).astype(np.uint32)


@pytest.mark.parametrize("left,right,clique", [
    (900, 400, 100),     # tails of up to four rows
    (900, 404, 100),     # a few past them
    (1200, 1000, 40),    # most past them
    (600, 1000, 33),
    (1000, 300, 250),    # none
    (700, 700, 2),       # rows of one entry
])
def test_long_tails(left, right, clique):
    torch = pytest.importorskip("torch")
    n, u, v = _core(left, right, clique)
    assert len(u) > 1 << 17
    src, dst = both_directions(u, v)
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    keep = torch.empty(len(src), dtype=torch.uint8, device="cuda")
    triangles = set()
    for limit in (None, 0):
        eng.set_list_limit(limit)
        for group in (0, 8, 32):
            eng.set_schedule(group, 32, 85, 50, 0)
            out.fill_(-1)
            torch.cuda.synchronize()
            eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, out.data_ptr())
            assert np.array_equal(out.cpu().numpy().view(np.uint32), ref["truss"]), (limit, group)
            triangles.add(eng.stats().triangles)
    for k in (3, 4, ref["k_max"]):
        eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, keep.data_ptr())
        assert np.array_equal(keep.cpu().numpy(), (ref["truss"] >= k).astype(np.uint8))
    assert len(triangles) == 1
    eng.close()
