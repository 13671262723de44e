"""The tiled builder reads an input error behind all of its launches: a refused input leaves the three outputs
alone, chained (small) or not, and the engine goes on working."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries,n,T", [(1, 2, 1), (2000, 100, 3), (400000, 5000, 4)])
def test_outputs_of_a_refused_input(entries, n, T):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(entries)
    src, dst = rng.integers(0, n, (2, entries)).astype(np.uint32)
    ptr, s, d = oracle.tiled_coocsr(n, src, dst, T)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()
    outs = [torch.full((size,), 77, dtype=torch.int32, device="cuda") for size in (len(ptr), entries, entries)]
    eng = kt.Engine(0)

    def call(a, b):
        torch.cuda.synchronize()
        eng.tiled_coocsr(a.data_ptr(), b.data_ptr(), entries, n, T, *(o.data_ptr() for o in outs))

    bad = dst.copy()
    bad[entries // 2] = n
    with pytest.raises(kt.KtrussError) as ei:
        call(dev(src), dev(bad))
    assert ei.value.status == 1 and all(bool((o == 77).all()) for o in outs)
    call(dev(src), dev(dst))
    for o, want in zip(outs, (ptr, s, d)):
        assert np.array_equal(o.cpu().numpy().view(np.uint32), want)
    eng.close()
