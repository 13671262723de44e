"""Small graphs' kernels are chained (each starts in its predecessor's tail): calls of alternating graphs,
one straight after the other, on both sides of the sizes up to which they are, and their replays."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu

LINE = 1 << 18  # entries, and vertices


def _graph(n, edges, seed):
    """`edges` distinct edges over n vertices, a third of them in a small core."""
    rng = np.random.default_rng([n, edges, seed])
    core = max(4, int((edges // 3) ** 0.5 * 1.7))
    ids = rng.choice(n, min(core, n), replace=False)
    a = np.concatenate([ids[rng.integers(0, len(ids), 2 * edges)], rng.integers(0, n, 2 * edges)])
    b = np.concatenate([ids[rng.integers(0, len(ids), 2 * edges)], rng.integers(0, n, 2 * edges)])
    keys = np.unique(np.minimum(a, b).astype(np.uint64) << np.uint64(32) | np.maximum(a, b).astype(np.uint64))
    keys = keys[(keys >> np.uint64(32)) != (keys & np.uint64(0xffffffff))]
    keys = np.sort(rng.choice(keys, edges, replace=False))
    src, dst = both_directions((keys >> np.uint64(32)).astype(np.uint32),
                               (keys & np.uint64(0xffffffff)).astype(np.uint32))
    order = rng.permutation(len(src))
    return n, src[order], dst[order]


@pytest.mark.parametrize("shapes", [
    [(40, 60), (3000, 9000), (LINE, 500), (LINE + 1, 500)],
    [(5000, LINE // 2), (5000, LINE // 2 + 1), (700, 4000)],
])
def test_alternating_graphs(shapes):
    torch = pytest.importorskip("torch")
    eng = kt.Engine(0)
    jobs = []
    for i, (n, edges) in enumerate(shapes):
        n, src, dst = _graph(n, edges, i)
        d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst)]
        truss = torch.zeros(len(src), dtype=torch.int32, device="cuda")
        keep = torch.zeros(len(src), dtype=torch.uint8, device="cuda")
        jobs.append((n, src, dst, d, truss, keep, oracle.decompose(n, src, dst, method="peel")["truss"]))
    torch.cuda.synchronize()
    for turn in range(12):
        for n, src, dst, (s, d), truss, keep, want in jobs:
            truss.fill_(-1)
            keep.fill_(7)
            torch.cuda.synchronize()
            k = 3 + turn % 3
            eng.ktruss(s.data_ptr(), d.data_ptr(), len(src), n, k, keep.data_ptr())
            eng.decompose(s.data_ptr(), d.data_ptr(), len(src), n, truss.data_ptr())
            if turn % 4 == 3:
                truss.fill_(-1)
                torch.cuda.synchronize()
                for _ in range(3):
                    eng.replay()
            assert np.array_equal(truss.cpu().numpy().view(np.uint32), want), (turn, n)
            assert np.array_equal(keep.cpu().numpy() == 1, want >= k), (turn, n, k)
    eng.close()
