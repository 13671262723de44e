"""A refused batch leaves both outputs alone, whatever its size: the input error is read only after the
kernels that write them are launched."""
import numpy as np
import pytest

import ktruss_gb300 as kt
from conftest import both_directions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [300, 6000, 40000])  # around 32,768 edges the host reads the error sooner
@pytest.mark.parametrize("what,status", [("bad vertex", 1), ("self loop", 2), ("duplicate", 3), ("asymmetric", 3)])
def test_outputs_of_a_refused_batch(size, what, status):
    torch = pytest.importorskip("torch")
    parts = [kt.gen_ba(size, 4, 9), kt.gen_ba(size // 2, 4, 10)]
    off = np.array([0, parts[0][0], parts[0][0] + parts[1][0]], np.uint32)
    u, v = (np.concatenate([parts[0][i], parts[1][i] + off[1]]) for i in (1, 2))
    src, dst = both_directions(u, v)
    i = len(src) // 3
    if what == "bad vertex":
        dst[i] = off[2] + 7
    elif what == "self loop":
        src[i] = dst[i]
    elif what == "duplicate":
        half = len(src) // 2
        src[0], dst[0], src[half], dst[half] = src[i], dst[i], dst[i], src[i]
    else:
        dst[i] = next(x for x in range(off[1]) if x != src[i] and x != dst[i])
    eng = kt.Engine(0)
    d_src, d_dst, d_off = (torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst, off))
    truss = torch.full((len(src),), 77, dtype=torch.int32, device="cuda")
    k_max = torch.full((2,), 77, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(kt.KtrussError) as ei:
        eng.decompose_batch(d_src.data_ptr(), d_dst.data_ptr(), len(src), int(off[2]), d_off.data_ptr(), 2,
                            truss.data_ptr(), k_max.data_ptr())
    assert ei.value.status == status
    assert bool((truss == 77).all()) and bool((k_max == 77).all())
    eng.close()
