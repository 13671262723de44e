"""Graphs without vertices or without edges on an engine that has done nothing else: every call finds a
workspace and gives the empty result, and the engine goes on working."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _calls(torch):
    off = torch.zeros(4, dtype=torch.int32, device="cuda")  # three graphs without vertices
    k_max = torch.full((3,), 77, dtype=torch.int32, device="cuda")
    sel = kt.Selector(0, seed=1)

    def decompose(e, n):
        e.decompose(0, 0, 0, n, 0, k_max.data_ptr())
        assert k_max.cpu().tolist() == [0, 77, 77]

    def batch(e, n):
        off[3] = n
        torch.cuda.synchronize()
        e.decompose_batch(0, 0, 0, n, off.data_ptr(), 3, 0, k_max.data_ptr())
        assert k_max.cpu().tolist() == [0, 0, 0]

    def selected(e, n):
        e.set_selector(sel)
        decompose(e, n)
        e.set_selector(None)

    return {
        "decompose": decompose,
        "selected": selected,
        "batch": batch,
        "ktruss": lambda e, n: e.ktruss(0, 0, 0, n, 4, 0),
        "ktruss_undirected": lambda e, n: (e.set_variant(directedness="undirected"), e.ktruss(0, 0, 0, n, 4, 0)),
        "features": lambda e, n: e.features(0, 0, 0, n),
        "autotune": lambda e, n: e.autotune(0, 0, 0, n, candidates=[(8, 32, 85, 50, 0)]),
        "noalloc": lambda e, n: (kt.decompose_noalloc(0, 0, 0, n, 0, k_max.data_ptr()), k_max.cpu().tolist()),
    }


@pytest.mark.parametrize("n", [0, 1, 5])
@pytest.mark.parametrize("name", ["decompose", "selected", "batch", "ktruss", "ktruss_undirected", "features",
                                  "autotune", "noalloc"])
def test_empty_graph_on_a_new_engine(name, n):
    torch = pytest.importorskip("torch")
    calls = _calls(torch)
    torch.cuda.synchronize()
    eng = kt.Engine(0)
    calls[name](eng, n)
    if name != "noalloc":
        st = eng.stats()
        assert st.num_edges == 0 and st.k_max == 0 and st.triangles == 0
    # the same engine on a graph with edges
    gn, u, v = kt.plant_cliques(*kt.gen_ba(300, 3, 5), 1, 9, 9, 6)
    src, dst = both_directions(u, v)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    out = torch.zeros(len(src), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), gn, out.data_ptr())
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.decompose(gn, src, dst, method="peel")["truss"])
    eng.close()
