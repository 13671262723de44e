"""The radix sort at the edges of its large tiles (6,144 keys), with and without values: all digits equal,
few keys a digit, and a last tile of one key."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions, edge_keys

pytestmark = pytest.mark.gpu

TILE = 6144
SIZES = [(1 << 18) + 1, 43 * TILE - 1, 43 * TILE, 43 * TILE + 1, 50 * TILE + TILE // 2, 51 * TILE - 31]


def _cuda(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()


@pytest.mark.parametrize("entries", SIZES)
@pytest.mark.parametrize("n", [2, 700, 1 << 20])
def test_keys(entries, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng([entries, n])
    src, dst = rng.integers(0, n, (2, entries)).astype(np.uint32)
    eng = kt.Engine(0)
    out = torch.zeros((2, 2 * entries), dtype=torch.int32, device="cuda")
    d_src, d_dst = _cuda(torch, src), _cuda(torch, dst)
    torch.cuda.synchronize()
    made = eng.symmetrize(d_src.data_ptr(), d_dst.data_ptr(), entries, n, out[0].data_ptr(), out[1].data_ptr(),
                          2 * entries)
    got = out.cpu().numpy().view(np.uint32)[:, :made].astype(np.uint64)
    want = edge_keys(src[src != dst], dst[src != dst])
    assert made == 2 * len(want)
    assert np.array_equal(got[0, : len(want)] << np.uint64(32) | got[1, : len(want)], want)
    eng.close()


@pytest.mark.parametrize("entries", [43 * TILE, 43 * TILE + 2, 50 * TILE + TILE // 2, 51 * TILE - 32])
def test_keys_with_values(entries):
    torch = pytest.importorskip("torch")
    n, u, v = kt.gen_rmat(14, 16, 0.57, 0.19, 0.19, 2)
    pick = np.random.default_rng(entries).choice(len(u), entries // 2, replace=False)
    src, dst = both_directions(u[pick], v[pick])
    order = np.random.default_rng(entries + 1).permutation(len(src))
    src, dst = src[order], dst[order]
    eng = kt.Engine(0)
    d_src, d_dst = _cuda(torch, src), _cuda(torch, dst)
    d_out = torch.zeros(len(src), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_out.data_ptr())
    ref = oracle.decompose(n, src, dst, method="peel")
    assert np.array_equal(d_out.cpu().numpy().view(np.uint32), ref["truss"])
    eng.close()
