"""Each kind of device wait, made to run out: it gives up within its limit, what comes behind it writes
nothing, and the engine's next calls are right."""
import time

import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("used", [False, True])
@pytest.mark.parametrize("wait", ["grid barrier", "list barrier", "look-back"])
def test_a_wait_that_runs_out(wait, used):
    torch = pytest.importorskip("torch")
    n, u, v = kt.gen_rmat(12, 12, 0.57, 0.19, 0.19, 3)
    src, dst = both_directions(u, v)
    want = oracle.decompose(n, src, dst, method="peel")["truss"]
    d_src, d_dst = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst))
    out = torch.empty(len(src), dtype=torch.int32, device="cuda")
    eng = kt.Engine(0)

    def check(call):
        out.fill_(-1)
        torch.cuda.synchronize()
        call()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)

    def decompose():
        eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, out.data_ptr())

    if used:
        check(decompose)
    t = time.perf_counter()
    assert eng.selftest_wait_timeout(wait, 20_000_000) == 11  # KT_ERR_TIMEOUT after 20 ms
    assert time.perf_counter() - t < 2
    if used:
        check(eng.replay)
    check(decompose)
    eng.set_wait_limit(1_000_000, 8)  # a limit for calls of this size
    check(decompose)
    check(eng.replay)
    eng.close()


def test_unknown_waits_are_refused():
    eng = kt.Engine(0)
    for wait, ns in ((3, 1000), (-1, 1000), (2, 0), (1, 6_000_000_000)):
        assert kt.lib().kt_engine_selftest_wait_timeout(eng._h, wait, ns) == 1  # KT_ERR_INVALID_ARG
    eng.close()
