"""Single-k queries whose first round removes many edges of graphs with a hub: the rows are compacted, but for
the hub's, which is longer than what a block compacts."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _wheel(rim, more):
    """A hub joined to a cycle, whose every `more`-th vertex has two more neighbours on it."""
    i = np.arange(1, rim + 1)
    j = i[::more]
    u = np.concatenate([np.zeros(rim, np.int64), i, j, j])
    v = np.concatenate([i, i % rim + 1, (j + 1) % rim + 1, (j + 2) % rim + 1])
    keys = np.unique(np.minimum(u, v) * (rim + 1) + np.maximum(u, v))
    return rim + 1, (keys // (rim + 1)).astype(np.uint32), (keys % (rim + 1)).astype(np.uint32)


@pytest.mark.parametrize("rim", [32000, 33500, 300000, 700000])  # around the longest row compacted; first rounds
@pytest.mark.parametrize("more", [2, 5, 1000])                   # packed from 2^19 edges on
def test_wheels(rim, more):
    torch = pytest.importorskip("torch")
    n, u, v = _wheel(rim, more)
    src, dst = both_directions(u, v)
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    keep = torch.empty(len(src), dtype=torch.uint8, device="cuda")
    for sched in ((8, 32, 85, 50, 0), (8, 8, 99, 10, 2), (8, 32, 0, 0, 0)):
        eng.set_schedule(*sched)
        for k in range(3, ref["k_max"] + 2):
            keep.fill_(7)
            torch.cuda.synchronize()
            eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, keep.data_ptr())
            assert np.array_equal(keep.cpu().numpy(), (ref["truss"] >= k).astype(np.uint8)), (sched, k)
    eng.close()
