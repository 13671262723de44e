"""A single-k call's first round run by the support count over the packed survivors (graphs of 2^19 edges
or more whose first frontier holds the schedule's recount share) against the walking rounds and
the oracle: the same edges kept, the same rounds."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions, edge_keys

pytestmark = pytest.mark.gpu


def _graph(edges, isolated, seed=4):
    n, u, v = kt.gen_rmat(16, 24, 0.57, 0.19, 0.19, seed)
    assert len(u) > edges
    pick = np.sort(np.random.default_rng(seed).choice(len(u), edges, replace=False))
    # vertices without edges at the end and between the others
    return 2 * n + isolated, *both_directions(2 * u[pick] + isolated, 2 * v[pick] + isolated)


def _run(torch, eng, n, src, dst, k, percent, replay=False):
    eng.set_schedule(8, 32, 85, percent)
    d_src, d_dst = (torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda() for a in (src, dst))
    d_keep = torch.full((len(src),), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, d_keep.data_ptr())
    if replay:
        d_keep.fill_(7)
        torch.cuda.synchronize()
        eng.replay()
    st, log = eng.stats(), eng.round_log()
    return d_keep.cpu().numpy(), list(log["size"]), st


@pytest.mark.parametrize("orientation", ["directed-by-degree", "directed-by-index"])
@pytest.mark.parametrize("edges,isolated", [(1 << 19, 0), (129 * 4096 - 1, 0), (129 * 4096 + 1, 1), (1 << 20, 3)])
def test_first_round_recounted(edges, isolated, orientation):
    torch = pytest.importorskip("torch")
    n, src, dst = _graph(edges, isolated)
    eng = kt.Engine(0)
    eng.set_variant(directedness=orientation)
    for k in (3, 4, 9, 30, 4000):
        walked, sizes, st = _run(torch, eng, n, src, dst, k, 0)
        assert st.num_rounds == len(sizes) and sum(sizes) == edges - int(walked.sum()) // 2
        if orientation == "directed-by-degree":
            want = edge_keys(*oracle.ktruss(n, src, dst, k))
            assert np.array_equal(edge_keys(src[walked == 1], dst[walked == 1]), want)
        share = 100 * sizes[0] // edges if sizes else 0
        lines = {share, share + 1, share * 10 // 7, share * 10 // 7 + 1, share * 10 // 7 + 2, 1, 50, 100}
        for percent in sorted({min(max(p, 1), 100) for p in lines}):  # on both sides of the line
            keep, s, t = _run(torch, eng, n, src, dst, k, percent)
            assert np.array_equal(keep, walked) and s == sizes, (k, percent)
            assert (t.num_rounds, t.triangles) == (st.num_rounds, st.triangles)
        keep, s, t = _run(torch, eng, n, src, dst, k, 1, replay=True)
        assert np.array_equal(keep, walked) and s == sizes
    eng.close()
