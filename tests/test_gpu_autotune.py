"""The autotuner on both peels: from triangle lists only the support group acts, so candidates that differ in
nothing else have one time and the engine's other settings stay; walking rows, every candidate is timed."""
import numpy as np
import pytest

import ktruss_gb300 as kt
from conftest import both_directions

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    torch = pytest.importorskip("torch")
    n, u, v = kt.gen_rmat(14, 16, 0.57, 0.19, 0.19, 3)
    src, dst = both_directions(u, v)
    d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst)]
    torch.cuda.synchronize()
    return d, len(src), n


@pytest.mark.parametrize("own", [(8, 32, 85, 50, 0), (4, 16, 0, 0, 0), (8, 16, 70, 20, 2)])
def test_lists_keep_the_other_settings(graph, own):
    (src, dst), N, n = graph
    eng = kt.Engine(0)
    eng.set_schedule(*own)
    best, table = eng.autotune(src.data_ptr(), dst.data_ptr(), N, n)
    times = {}
    for s, ms in table:
        assert ms > 0 and times.setdefault(s.support_group, ms) == ms
    assert len(times) == 3 and times[best.support_group] == min(times.values())
    assert eng.schedule().as_tuple() == best.as_tuple()
    group = [s.as_tuple() for s, _ in table if s.support_group == best.support_group]
    kept = (best.support_group, *own[1:])
    assert best.as_tuple() == (kept if kept in group else group[0])
    eng.close()


def test_walks_are_timed_one_by_one(graph):
    (src, dst), N, n = graph
    eng = kt.Engine(0)
    eng.set_list_limit(0)
    best, table = eng.autotune(src.data_ptr(), dst.data_ptr(), N, n)
    assert len({ms for _, ms in table}) > 3
    assert best.as_tuple() == min(table, key=lambda x: x[1])[0].as_tuple() == eng.schedule().as_tuple()
    eng.close()


def test_an_invalid_candidate_leaves_the_schedule(graph):
    (src, dst), N, n = graph
    eng = kt.Engine(0)
    eng.set_schedule(16, 8, 0, 0, 1)
    with pytest.raises(kt.KtrussError) as ei:
        eng.autotune(src.data_ptr(), dst.data_ptr(), N, n, candidates=[(8, 32, 85, 50, 0), (8, 32, 85, 50, 3)])
    assert ei.value.status == 1 and eng.schedule().as_tuple() == (16, 8, 0, 0, 1)
    eng.close()
