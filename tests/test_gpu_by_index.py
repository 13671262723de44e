"""Support counts of graphs oriented by vertex id, where hubs have long rows and tails: on both sides of the
lines that choose how an edge is counted, with both support schedules and after a packed first round, whose
rows are in no order of length."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _shuffled(n, u, v):
    p = np.random.default_rng(1).permutation(n)
    a, b = p[u], p[v]
    return n, np.minimum(a, b).astype(np.uint32), np.maximum(a, b).astype(np.uint32)


def _hub_tails(hubs, n):
    """Hubs with the smallest ids, next to each other and to all others: tails of thousands over rows of 40."""
    u, v = np.triu_indices(hubs, 1, n)
    ring = np.arange(hubs, n)
    us, vs = [u], [v]
    for step in range(1, 41):
        us.append(ring[:-step])
        vs.append(ring[step:])
    return n, np.concatenate(us).astype(np.uint32), np.concatenate(vs).astype(np.uint32)


GRAPHS = {
    "rmat15": lambda: kt.gen_rmat(15, 16, 0.57, 0.19, 0.19, 3),          # edge-centric by its size
    "rmat16_more": lambda: kt.gen_rmat(16, 20, 0.57, 0.19, 0.19, 4),     # past it, hubs first
    "rmat16_shuffled": lambda: _shuffled(*kt.gen_rmat(16, 20, 0.57, 0.19, 0.19, 4)),
    "er1500": lambda: kt.gen_er(1500, 0.3, 5),                           # small, but 450 neighbours a vertex
    "hub_tails": lambda: _hub_tails(70, 9000),
    "sparse": lambda: kt.gen_er(300000, 2e-5, 6),                        # six neighbours a vertex
    # a first round that removes all edges, or all but a clique, from rows of a few entries in no order
    "tree": lambda: (800001, (np.arange(1, 800001) // 4).astype(np.uint32), np.arange(1, 800001, dtype=np.uint32)),
    "tree_clique": lambda: kt.plant_cliques(600001, (np.arange(1, 600001) // 4).astype(np.uint32),
                                            np.arange(1, 600001, dtype=np.uint32), 2, 12, 30, 7),
}


@pytest.mark.parametrize("name", GRAPHS)
def test_by_index_counts(name):
    torch = pytest.importorskip("torch")
    n, u, v = GRAPHS[name]()
    assert len(u) > 1 << 18
    src, dst = both_directions(u, v)
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    keep = torch.empty(len(src), dtype=torch.uint8, device="cuda")
    triangles = set()
    for directedness in ("directed-by-degree", "directed-by-index"):
        eng.set_variant(directedness=directedness)
        for group in (0, 8):
            eng.set_schedule(group, 32, 85, 50, 0)
            for k in (3, 4, max(5, ref["k_max"] // 2), ref["k_max"]):
                keep.fill_(7)
                torch.cuda.synchronize()
                eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, keep.data_ptr())
                want = (ref["truss"] >= k).astype(np.uint8)
                assert np.array_equal(keep.cpu().numpy(), want), (directedness, group, k)
                triangles.add(eng.stats().triangles)
    assert len(triangles) == 1
    eng.close()


def test_first_rounds_below_the_recount_share():
    """A first round of seven tenths of the recount share or more is counted again over the packed survivors by
    degree, and walked by vertex id, where counting costs more; from the share on both are packed."""
    torch = pytest.importorskip("torch")
    n, u, v = kt.gen_rmat(16, 24, 0.57, 0.19, 0.19, 4)
    u, v = u[: 1 << 20], v[: 1 << 20]
    src, dst = both_directions(u, v)
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).cuda() for x in (src, dst))
    keep = torch.empty(len(src), dtype=torch.uint8, device="cuda")
    got = {}
    for directedness in ("directed-by-degree", "directed-by-index"):
        eng.set_variant(directedness=directedness)
        eng.set_schedule(8, 32, 85, 0)
        eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, 12, keep.data_ptr())
        want = keep.cpu().numpy()
        share = 100 * int(eng.round_log()["size"][0]) // len(u)
        assert 5 < share < 90
        for percent in (share, share + 1, share * 10 // 7 - 1, min(100, share * 10 // 7 + 2)):
            eng.set_schedule(8, 32, 85, percent)
            keep.fill_(7)
            torch.cuda.synchronize()
            eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, 12, keep.data_ptr())
            assert np.array_equal(keep.cpu().numpy(), want)
            got[directedness, percent > share, percent * 7 // 10 > share] = eng.stats().peel_phase_ms[4] > 0
    # peel_phase_ms[4]: time in rounds that count again
    assert got["directed-by-degree", False, False] and got["directed-by-index", False, False]
    assert got["directed-by-degree", True, False] and not got["directed-by-index", True, False]
    assert not got["directed-by-degree", True, True] and not got["directed-by-index", True, True]
    eng.close()
