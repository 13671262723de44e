"""The walking peel in decompositions, which take triangle lists unless these are switched off, too many or
too large: every schedule, chunks past the end of their buffer, batches and replays, with no memory for lists
and on graphs that walk by themselves."""
import itertools

import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu

GRAPHS = {
    "rmat13": lambda: kt.gen_rmat(13, 16, 0.57, 0.19, 0.19, 11),
    "ba6000_cliques": lambda: kt.plant_cliques(*kt.gen_ba(6000, 4, 12), 3, 16, 48, 13),
    "ws8000": lambda: kt.gen_ws(8000, 10, 0.1, 14),
}
SCHEDULES = list(itertools.product((0, 8), (8, 16, 32), (0, 50, 85), (0, 1, 50), (0, 1, 2)))


class Run:
    """A graph on the device and an engine without lists (or, with_lists, one as users have it)."""

    def __init__(self, n, u, v, with_lists=False):
        self.torch = pytest.importorskip("torch")
        self.n, (src, dst) = n, both_directions(u, v)
        self.N = len(src)
        self.want = oracle.decompose(n, src, dst, method="peel")
        self.eng = kt.Engine(0)
        if not with_lists:
            self.eng.set_list_limit(0)
        self.eng.reserve(n, self.N)
        self.src, self.dst = (self.torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
        self.out = self.torch.empty(self.N, dtype=self.torch.int32, device="cuda")
        self.k_max = self.torch.zeros(1, dtype=self.torch.int32, device="cuda")

    def decompose(self):
        self.eng.decompose(self.src.data_ptr(), self.dst.data_ptr(), self.N, self.n, self.out.data_ptr(),
                           self.k_max.data_ptr())

    def check(self, call):
        self.out.fill_(-1)
        self.torch.cuda.synchronize()
        call()
        assert np.array_equal(self.out.cpu().numpy().view(np.uint32), self.want["truss"])
        assert int(self.k_max.item()) == self.want["k_max"]
        st = self.eng.stats()
        assert st.walk_entries != 3 * st.triangles  # lists queue exactly these
        return st


@pytest.mark.parametrize("name", GRAPHS)
def test_every_schedule_walks(name):
    run = Run(*GRAPHS[name]())
    for sched in SCHEDULES:
        run.eng.set_schedule(*sched)
        st = run.check(run.decompose)
        assert (st.compactions > 0) == (sched[2] != 0), sched


def test_replayed_walks():
    run = Run(*GRAPHS["ba6000_cliques"]())
    run.check(run.decompose)
    for sched in ((8, 32, 85, 50, 0), (16, 8, 0, 0, 1), (4, 16, 85, 1, 2)):
        run.eng.set_schedule(*sched)
        run.check(run.eng.replay)
        run.check(run.eng.replay)


@pytest.mark.parametrize("sched", [(4, 8, 50, 25, 2), (8, 32, 85, 0, 1)])
def test_batch_walks(sched):
    n, u, v, off = kt.gen_batch(24, 500, 4000, 31)
    run = Run(n, u, v)
    run.eng.set_schedule(*sched)
    d_off = run.torch.from_numpy(off.view(np.int32)).cuda()
    k_max = run.torch.zeros(len(off) - 1, dtype=run.torch.int32, device="cuda")
    run.k_max.fill_(run.want["k_max"])
    run.check(lambda: run.eng.decompose_batch(run.src.data_ptr(), run.dst.data_ptr(), run.N, n, d_off.data_ptr(),
                                              len(off) - 1, run.out.data_ptr(), k_max.data_ptr()))
    assert int(k_max.max()) == run.want["k_max"]


def _cliques(sizes):
    us, vs, base = [], [], 0
    for s in sizes:
        u, v = np.triu_indices(s, 1)
        us.append(u + base)
        vs.append(v + base)
        base += s
    return base, np.concatenate(us).astype(np.uint32), np.concatenate(vs).astype(np.uint32)


@pytest.mark.parametrize("w,rc,pb", [(8, 0, 0), (8, 0, 2), (8, 50, 2), (32, 0, 1)])
@pytest.mark.parametrize("sizes", [[20] * 300, [100, 100, 64]], ids=["many_small", "few_large"])
def test_chunks_past_their_buffer(sizes, w, rc, pb):
    """All edges of many cliques in one frontier: with narrow chunks more of them than the buffer's m + 4096;
    the rest is walked a warp (many edges) or a block (few edges) an edge."""
    n, u, v = _cliques(sizes)
    if w == 8:
        assert sum(s * (s - 1) // 2 * -(-(s - 1) // w) for s in sizes) > len(u) + 4096
    run = Run(n, u, v)
    run.eng.set_schedule(8, w, 85, rc, pb)
    run.check(run.decompose)


@pytest.mark.parametrize("name,make", [
    ("near-cliques", lambda: _cliques([64] * 140)),          # 282,240 edges: width 8 overflows the buffer
    ("dense", lambda: kt.gen_er(900, 0.9, 3)),               # more than 512 list entries an edge
])
@pytest.mark.parametrize("sched", [(8, 8, 85, 0, 0), (8, 32, 0, 1, 2), (8, 32, 85, 50, 0)])
def test_graphs_that_walk_by_themselves(name, make, sched):
    run = Run(*make(), with_lists=True)
    run.eng.set_schedule(*sched)
    run.check(run.decompose)
    run.check(run.eng.replay)
