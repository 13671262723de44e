"""The one-pass scans and radix passes of the CSR build at the edges of their tiles (1,024 keys up to
2^18, 4,096 above), and rows that have no entries, in front (ranks by degree) and in between
(orientation by vertex id)."""
import numpy as np
import pytest

import ktruss_gb300 as kt
import oracle
from conftest import both_directions, edge_keys

pytestmark = pytest.mark.gpu


def _cuda(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()


@pytest.mark.parametrize("entries", [1, 2, 31, 1023, 1024, 1025, 4095, 4096, 4097, (1 << 18) - 1, 1 << 18,
                                     (1 << 18) + 1, 64 * 4096 + 4095, 300 * 4096 + 1])
@pytest.mark.parametrize("bits", [1, 8, 9, 17])
def test_sort_at_tile_edges(entries, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng([entries, bits])
    n = (1 << bits) - (bits > 1)
    src, dst = rng.integers(0, n, (2, entries)).astype(np.uint32)
    if entries > 4:  # runs of equal keys as well
        src[: entries // 3], dst[: entries // 3] = 0, n - 1
    eng = kt.Engine(0)
    out = torch.zeros((2, 2 * entries), dtype=torch.int32, device="cuda")
    d_src, d_dst = _cuda(torch, src), _cuda(torch, dst)
    torch.cuda.synchronize()
    made = eng.symmetrize(d_src.data_ptr(), d_dst.data_ptr(), entries, n, out[0].data_ptr(), out[1].data_ptr(),
                          2 * entries)
    want = edge_keys(src[src != dst], dst[src != dst])
    got = out.cpu().numpy().view(np.uint32)[:, :made].astype(np.uint64)
    u = made // 2
    assert u == len(want)
    assert np.array_equal(got[0, :u] << np.uint64(32) | got[1, :u], want)
    assert np.array_equal(got[0, u:], got[1, :u]) and np.array_equal(got[1, u:], got[0, :u])
    eng.close()


def _spread(n, u, v, factor):
    """The graph with `factor` - 1 isolated vertices after each vertex."""
    return n * factor + 5, (u * factor + 2).astype(np.uint32), (v * factor + 2).astype(np.uint32)


@pytest.mark.parametrize("factor", [1, 3, 50])
@pytest.mark.parametrize("size", [5, 1100, 5000])
def test_rows_without_entries(factor, size):
    torch = pytest.importorskip("torch")
    n, u, v = _spread(*kt.plant_cliques(*kt.gen_ba(size, 3, 5), 1, 5, 5, 6), factor)
    src, dst = both_directions(u, v)
    order = np.random.default_rng(7).permutation(len(src))
    src, dst = src[order], dst[order]
    ref = oracle.decompose(n, src, dst, method="peel")
    eng = kt.Engine(0)
    d_src, d_dst = _cuda(torch, src), _cuda(torch, dst)
    d_out = torch.zeros(len(src), dtype=torch.int32, device="cuda")
    keep = torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    eng.decompose(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, d_out.data_ptr())
    assert np.array_equal(d_out.cpu().numpy().view(np.uint32), ref["truss"])
    for directedness in ("directed-by-degree", "directed-by-index"):
        eng.set_variant(directedness=directedness)
        for k in (3, 4, 5):
            eng.ktruss(d_src.data_ptr(), d_dst.data_ptr(), len(src), n, k, keep.data_ptr())
            assert np.array_equal(keep.cpu().numpy().astype(bool), ref["truss"] >= k), (directedness, k)
    eng.close()


def _broken(src, dst, n, what):
    src, dst = src.copy(), dst.copy()
    i = len(src) // 3
    if what == "bad vertex":
        dst[i] = n + 7
    elif what == "self loop":
        src[i] = dst[i]
    elif what == "duplicate":  # both directions of an edge twice, another edge gone
        half = len(src) // 2
        src[0], dst[0], src[half], dst[half] = src[i], dst[i], dst[i], src[i]
    else:  # one direction missing, its slot filled with a new edge's one direction
        dst[i] = (dst[i] + 1) % n if (dst[i] + 1) % n != src[i] else (dst[i] + 2) % n
    return src, dst


@pytest.mark.parametrize("size", [300, 6000, 40000])
@pytest.mark.parametrize("what,status", [("bad vertex", 1), ("self loop", 2), ("duplicate", 3), ("asymmetric", 3)])
def test_refused_inputs(size, what, status):
    """Input errors are read once a call, after the kernels behind the build were launched: they are
    still the call's status, nothing is written, and the engine keeps working."""
    torch = pytest.importorskip("torch")
    n, u, v = kt.gen_ba(size, 8, 9)
    src, dst = both_directions(u, v)
    b_src, b_dst = _broken(src, dst, n, what)
    eng = kt.Engine(0)
    good = [_cuda(torch, x) for x in (src, dst)]
    bad = [_cuda(torch, x) for x in (b_src, b_dst)]
    truss = torch.full((len(src),), 77, dtype=torch.int32, device="cuda")
    keep = torch.full((len(src),), 77, dtype=torch.uint8, device="cuda")
    k_max = torch.full((1,), 77, dtype=torch.int32, device="cuda")
    off = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s, d = (x.data_ptr() for x in bad)
    calls = [lambda: eng.decompose(s, d, len(src), n, truss.data_ptr(), k_max.data_ptr()),
             lambda: eng.ktruss(s, d, len(src), n, 4, keep.data_ptr()),
             lambda: eng.decompose_batch(s, d, len(src), n, off.data_ptr(), 1, truss.data_ptr(), k_max.data_ptr())]
    if len(src) <= 1 << 19:
        calls.append(lambda: kt.decompose_noalloc(s, d, len(src), n, truss.data_ptr(), k_max.data_ptr()))
    for i, call in enumerate(calls):
        with pytest.raises(kt.KtrussError) as ei:
            call()
        assert ei.value.status == status, i
        assert bool((truss == 77).all()) and bool((keep == 77).all())
    eng.decompose(good[0].data_ptr(), good[1].data_ptr(), len(src), n, truss.data_ptr(), k_max.data_ptr())
    ref = oracle.decompose(n, src, dst, method="peel")
    assert np.array_equal(truss.cpu().numpy().view(np.uint32), ref["truss"]) and int(k_max.item()) == ref["k_max"]
    eng.close()
