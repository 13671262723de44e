"""The decomposition from triangle lists, bit for bit against the oracle where its kernel can go
wrong: rounds past the period of the state bytes' stamps, more queued edges than a block's queue
holds (at a level start and from decrements), lists of more chunks than the chunk buffer, the
smallest graphs, odd edge counts, and graphs on both sides of the density rule."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _union(parts):
    us, vs, base = [], [], 0
    for n, u, v in parts:
        us.append(np.asarray(u, np.int64) + base)
        vs.append(np.asarray(v, np.int64) + base)
        base += n
    return base, np.concatenate(us).astype(np.uint32), np.concatenate(vs).astype(np.uint32)


def _clique(s):
    u, v = np.triu_indices(s, 1)
    return s, u, v


def _strip(s):
    """A strip of triangles (i, i+1, i+2): level 4 eats it from both ends, one triangle a round."""
    i = np.arange(s - 1)
    return s, np.concatenate([i, i[:-1]]), np.concatenate([i + 1, i[:-1] + 2])


def _copies(part, count):
    n, u, v = (np.asarray(x) for x in part)
    at = (np.arange(count) * int(n))[:, None]
    return int(n) * count, (u + at).ravel(), (v + at).ravel()


def _core(r, c):
    """A complete bipartite graph of r + r vertices whose first c left vertices form a clique."""
    c = min(c, r)
    left, right = np.divmod(np.arange(r * r), r)
    cu, cv = np.triu_indices(c, 1)
    return 2 * r, np.concatenate([left, cu]), np.concatenate([right + r, cv])


GRAPHS = {
    "one_edge": lambda: (2, np.array([0], np.uint32), np.array([1], np.uint32)),
    "one_triangle": lambda: _union([_clique(3)]),
    "long_strip": lambda: _union([_strip(3001), _clique(6)]),          # 1,500 rounds in one level
    "strips_past_solo": lambda: _union([_copies(_strip(1203), 40), _clique(7)]),
    "many_cliques": lambda: _union([_copies(_clique(5), 90000), _clique(6)]),    # 900,000 edges at a level start
    "many_strips": lambda: _union([_copies(_strip(9), 220000), _clique(5)]),     # 900,000 edges queued in a round
    "chunk_overflow": lambda: _union([_copies(_clique(100), 25), _clique(120)]),  # four chunks an edge
    "rmat12_odd": lambda: kt.gen_rmat(12, 13, 0.57, 0.19, 0.19, 77),
    # the vertex-centric count and the three kernels of the fill: graphs of 2^18 edges and more
    "rmat15": lambda: kt.gen_rmat(15, 16, 0.57, 0.19, 0.19, 80),
    "rmat15_cliques": lambda: kt.plant_cliques(*kt.gen_rmat(15, 12, 0.45, 0.22, 0.22, 81), 12, 60, 200, 82),
    "rows_of_2000": lambda: _core(2000, 100),   # the longest rows that are hashed ...
    "rows_of_2100": lambda: _core(2100, 100),   # ... and rows that are not
    "rows_at_the_lines": lambda: _union([_core(r, c) for r in (31, 32, 127, 128, 129) for c in (20, 66)] +
                                        [_core(500, 70)]),
    "hubs": lambda: kt.plant_cliques(*kt.gen_ba(20000, 12, 78), 6, 30, 90, 79),
}


@pytest.mark.parametrize("name", GRAPHS)
def test_lists_match_oracle(name):
    torch = pytest.importorskip("torch")
    n, u, v = GRAPHS[name]()
    src, dst = both_directions(u, v)
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    eng.reserve(n, len(src))
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    d_out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    d_k = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):  # the second call finds the first one's lists and states in its workspace
        d_out.fill_(-1)
        torch.cuda.synchronize()
        eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_out.data_ptr(), d_k.data_ptr())
        assert int(d_k.item()) == ref["k_max"]
        assert np.array_equal(d_out.cpu().numpy().view(np.uint32), ref["truss"])
    st = eng.stats()
    assert st.num_levels <= ref["k_max"] and st.compactions == 0
    eng.close()


@pytest.mark.parametrize("s", [190, 230])
def test_density_rule(s):
    """Cliques below and above the list entries per edge at which the rows are walked instead."""
    torch = pytest.importorskip("torch")
    n, u, v = _union([_clique(s), _clique(s - 7)])
    src, dst = both_directions(u, v)
    eng = kt.Engine(0)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    d_out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_out.data_ptr())
    first = s * (s - 1) // 2
    want = np.where(np.arange(len(u)) < first, s, s - 7)
    assert np.array_equal(d_out.cpu().numpy(), np.concatenate([want, want]))
    eng.close()
