"""The device memory of the triangle lists: bounded and given back on demand, given back by itself when the
engine needs the memory for another of its arrays, and never allocated behind a reservation with limit 0."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


def _device(torch, n, u, v):
    src, dst = both_directions(u, v)
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    return dict(n=n, N=len(src), src=d_src, dst=d_dst, out=torch.empty(len(src), dtype=torch.int32, device="cuda"),
                want=oracle.decompose(n, src, dst, method="peel")["truss"])


def _check(torch, eng, g, lists, run=None):
    """One call (or `run`), its result, and whether it went from lists: these queue three entries a triangle."""
    g["out"].fill_(-1)
    torch.cuda.synchronize()
    if run:
        run()
    else:
        eng.decompose(g["src"].data_ptr(), g["dst"].data_ptr(), g["N"], g["n"], g["out"].data_ptr())
    assert np.array_equal(g["out"].cpu().numpy().view(np.uint32), g["want"])
    st = eng.stats()
    assert (st.walk_entries == 3 * st.triangles) == lists
    return st.triangles


GRAPHS = {"small": lambda: kt.gen_rmat(11, 12, 0.57, 0.19, 0.19, 3),   # lists without a count
          "counted": lambda: kt.gen_rmat(13, 16, 0.57, 0.19, 0.19, 4),
          "large": lambda: kt.gen_rmat(15, 16, 0.57, 0.19, 0.19, 5)}


@pytest.mark.parametrize("name", GRAPHS)
def test_limits(name):
    torch = pytest.importorskip("torch")
    g = _device(torch, *GRAPHS[name]())
    eng = kt.Engine(0)
    eng.reserve(g["n"], g["N"])
    limit, held = eng.list_limit()
    assert limit is None and 0 < held < 68_000_000
    need = 24 * _check(torch, eng, g, True)
    held = eng.list_limit()[1]
    assert held >= need
    eng.replay()
    eng.set_list_limit(0)  # the replay that was captured with them does without
    assert eng.list_limit() == (0, 0)
    _check(torch, eng, g, False, eng.replay)
    _check(torch, eng, g, False)
    _check(torch, eng, g, False, eng.replay)
    eng.set_list_limit(need - 1)  # (a small graph is counted when the buffer for all of its size does not fit)
    _check(torch, eng, g, False)
    eng.set_list_limit(need)
    _check(torch, eng, g, True)
    assert need <= eng.list_limit()[1] <= need + 8
    eng.set_list_limit()
    _check(torch, eng, g, True)
    _check(torch, eng, g, True, eng.replay)
    eng.close()


def test_no_allocation_behind_a_reservation():
    torch = pytest.importorskip("torch")
    graphs = [_device(torch, *GRAPHS[name]()) for name in GRAPHS]
    keep = torch.empty(max(g["N"] for g in graphs), dtype=torch.uint8, device="cuda")
    eng = kt.Engine(0)
    eng.set_list_limit(0)
    eng.reserve(max(g["n"] for g in graphs), max(g["N"] for g in graphs))
    for i in range(2):  # (the first calls load their kernels)
        if i:
            free = torch.cuda.mem_get_info()[0]
        for g in graphs:
            _check(torch, eng, g, False)
            eng.ktruss(g["src"].data_ptr(), g["dst"].data_ptr(), g["N"], g["n"], 4, keep.data_ptr())
            assert np.array_equal(keep[: g["N"]].cpu().numpy().astype(bool), g["want"] >= 4)
    assert torch.cuda.mem_get_info()[0] == free
    eng.close()


def test_a_reservation_takes_the_lists_memory():
    """With little memory left on the device the engine's own workspace takes the place of the lists."""
    torch = pytest.importorskip("torch")
    g = _device(torch, *kt.gen_er(900, 0.7, 3))  # 440 entries an edge
    eng = kt.Engine(0)
    eng.reserve(g["n"], g["N"])
    need = 24 * _check(torch, eng, g, True)
    torch.cuda.empty_cache()
    spare = 4 << 30
    block = (torch.cuda.mem_get_info()[0] - spare) // 4
    fill = [torch.empty(block, dtype=torch.uint8, device="cuda") for _ in range(4)]
    left = torch.cuda.mem_get_info()[0]
    # about 79 bytes an entry of workspace: more than what is left, less than it and the lists
    eng.reserve(g["n"], g["N"] + (left + need // 2) // 77)
    assert eng.list_limit()[1] < need
    del fill
    torch.cuda.empty_cache()
    _check(torch, eng, g, True)
    eng.close()


def test_limit_of_the_host_buffer_calls():
    n, u, v = GRAPHS["large"]()
    g = kt.COOGraph.from_undirected(n, u, v)
    want = kt.decompose(g)
    limit, held = kt.list_limit()
    st = kt.last_stats()
    assert limit is None and held >= 24 * st.triangles and st.walk_entries == 3 * st.triangles
    kt.set_list_limit(0)
    assert kt.list_limit() == (0, 0)
    got = kt.decompose(g)
    st = kt.last_stats()
    assert st.walk_entries != 3 * st.triangles
    kt.set_list_limit()
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]
