"""The calls that a user of this package makes, with the sizes they are made at.

A case names an operation and a graph.  Graphs are seeded: R-MAT, Watts-Strogatz and uniform random
ones are drawn on the GPU, Barabasi-Albert graphs and batches come from the package's generators.
Every undirected edge is listed in both directions, in one of three orders: "pairs" (all (u, v) in
sorted order, then all reversed, as COOGraph.from_undirected makes them), "rows" (sorted by source,
as adjacency files are) and "shuffled" (as edges arrive in a stream).

All outputs are whole numbers and bytes: there is nothing to compute in 64 bits, so no exact().
"""
import concurrent.futures
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ktruss-explorer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import ktruss_gb300 as kt  # noqa: E402

ORDERS = ("pairs", "rows", "shuffled")


def listed():
    return [
        # one k-truss query on a small social graph, as an interactive caller sends it: launches
        dict(name="query_ba2000", op="ktruss", k=4, family="ba", n=2000, edges=15_000, order="pairs"),
        # the complete decomposition of a small uniform graph: launches and round latency
        dict(name="decompose_er4096", op="decompose", family="er", n=4096, edges=32_000, order="pairs"),
        # a community graph read from an adjacency file: hundreds of short rounds
        dict(name="decompose_rmat16", op="decompose", family="rmat", n=1 << 16, edges=900_000, order="rows"),
        # the headline graph: a web or social graph of 15 M edges
        dict(name="decompose_rmat20", op="decompose", family="rmat", n=1 << 20, edges=15_000_000, order="pairs"),
        # the same family past the L2 cache
        dict(name="decompose_rmat22", op="decompose", family="rmat", n=1 << 22, edges=60_000_000, order="pairs"),
        # a mesh-like graph without hubs, its edges in no order: few levels, many edges in each
        dict(name="decompose_ws1m", op="decompose", family="ws", n=1000003, edges=9_950_000, order="shuffled"),
        # one single-k query on the headline graph, the unit that the reference times
        dict(name="query_rmat20_k3", op="ktruss", k=3, family="rmat", n=1 << 20, edges=15_000_000, order="pairs"),
        # a dense-core query: most edges go in the first rounds
        dict(name="query_rmat18_k32", op="ktruss", k=32, family="rmat", n=1 << 18, edges=3_700_000, order="rows"),
        # many small graphs in one call
        dict(name="batch256", op="batch", family="batch", graphs=256, n_min=500, n_max=50000, order="pairs"),
        # the host-buffer call of a program that keeps its graph in numpy arrays
        dict(name="host_rmat14", op="host", family="rmat", n=1 << 14, edges=220_000, order="rows"),
        # the text of a graph file, already on the device, into entries
        dict(name="parse_rmat18", op="parse", family="rmat", n=1 << 18, edges=3_700_000, order="rows"),
        # a raw edge stream (one direction, repeats, self loops) into the symmetric simple graph
        dict(name="symmetrize_rmat20", op="symmetrize", family="rmat", n=1 << 20, edges=1 << 24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scaled(rng, n_max, degree):
    """Vertices and edges of a graph with at most n_max vertices; n is rarely a round number."""
    n = _log(rng, 1500, n_max)
    return dict(n=n, edges=int(n * rng.uniform(*degree)))


def draw(rng):
    op = rng.choice(("decompose", "decompose", "ktruss", "ktruss", "batch", "host", "parse", "symmetrize"))
    if op == "batch":
        lo = _log(rng, 500, 2000)
        return dict(op=op, family="batch", graphs=_log(rng, 8, 256), n_min=lo, n_max=lo * rng.randint(2, 25), order="pairs")
    if op == "symmetrize":
        return dict(op=op, family="rmat", **_scaled(rng, 1 << 20, (4, 16)))
    if op == "parse":
        return dict(op=op, family="rmat", order=rng.choice(ORDERS), **_scaled(rng, 1 << 18, (4, 16)))
    if op == "host":
        return dict(op=op, family=rng.choice(("rmat", "er", "ws")), order=rng.choice(ORDERS), **_scaled(rng, 1 << 17, (4, 16)))
    family = rng.choice(("rmat", "rmat", "er", "ws", "ba"))
    case = dict(op=op, family=family, order=rng.choice(ORDERS),
                **_scaled(rng, 100000 if family == "ba" else 3 << 20, (4, 16) if family != "ba" else (2, 12)))
    if op == "ktruss":
        # up to the cores that graphs of the family and size have
        deepest = {"rmat": 5 if case["n"] < 20000 else 32, "ws": 5}.get(family, 3)
        case["k"] = rng.choice([k for k in (3, 3, 4, 5, 8, 16, 32) if k <= deepest])
    return case


# ---- graphs ---------------------------------------------------------------------------------

def _rmat(n, draws, gen):
    """R-MAT draws (0.57, 0.19, 0.19, 0.05) on ceil(log2 n) levels, ids folded into [0, n)."""
    u = torch.zeros(draws, dtype=torch.int64, device="cuda")
    v = torch.zeros(draws, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(draws, generator=gen, device="cuda")
        u = 2 * u + (r >= 0.76)
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return u % n, v % n


def _er(n, draws, gen):
    ends = torch.randint(0, n, (2, draws), generator=gen, device="cuda")
    return ends[0], ends[1]


def _ws(n, draws, gen):
    """A ring lattice with ceil(draws / n) neighbours on each side; a tenth of the edges rewired."""
    half = -(-draws // n)
    u = torch.arange(n, device="cuda").repeat_interleave(half)
    v = (u + 1 + torch.arange(half, device="cuda").repeat(n)) % n
    moved = torch.rand(n * half, generator=gen, device="cuda") < 0.1
    return u, torch.where(moved, torch.randint(0, n, (n * half,), generator=gen, device="cuda"), v)


def _ba(n, draws, gen):
    _, u, v = kt.gen_ba(n, -(-draws // n), _seed(gen))
    return (torch.from_numpy(x.astype(np.int64)).cuda() for x in (u, v))


def _seed(gen):
    return int(torch.randint(1, 1 << 30, (1,), generator=gen, device="cuda"))


def _thin(u, v, edges, gen):
    """`edges` of the listed edges, the others dropped at random, in the order they are listed."""
    at = torch.randperm(u.numel(), generator=gen, device="cuda")[:edges].sort().values
    return u[at], v[at]


def _simple(case, gen):
    """The case's number of distinct undirected edges (lower, higher), in sorted order."""
    n, edges, draws = case["n"], case["edges"], case["edges"]
    while True:
        draws += draws // 16 + 8
        u, v = {"rmat": _rmat, "er": _er, "ws": _ws, "ba": _ba}[case["family"]](n, draws, gen)
        keys = torch.unique((torch.minimum(u, v) * n + torch.maximum(u, v))[u != v])
        if keys.numel() >= edges:
            return _thin(keys // n, keys % n, edges, gen)


def _batch(case, gen):
    """Graphs of sizes spread over the logarithm of [n_min, n_max], Barabasi-Albert and
    Watts-Strogatz in turn, with up to three planted cliques each; one edge in twenty dropped."""
    G, lo, hi = case["graphs"], case["n_min"], case["n_max"]
    seed, off, nominal, make = _seed(gen), [0], 0, []
    for g in range(G):
        n = int(lo * (hi / lo) ** (g / max(1, G - 1)))
        half = ((2, 4, 8, 16), (3, 5, 10))[g % 2][g // 2 % (4 - g % 2)]
        size, count = min(n // 8, 8 + 13 * g % 57), g % 4
        off.append(off[-1] + n)
        nominal += n * half - half * half + count * size * (size - 1) // 2
        make.append((n, half, g % 2, count, size, seed + 2 * g))

    def one(a):
        n, half, ws, count, size, seed = a
        base = kt.gen_ws(n, 2 * half, 0.1, seed) if ws else kt.gen_ba(n, half, seed)
        return kt.plant_cliques(*base, count, size, size, seed + 1) if count else base

    with concurrent.futures.ThreadPoolExecutor(16) as pool:
        parts = list(pool.map(one, make))
    u, v = (torch.from_numpy(np.concatenate([p[i] + np.uint32(o) for p, o in zip(parts, off)]).astype(np.int64)).cuda()
            for i in (1, 2))
    edges = nominal * 19 // 20
    if u.numel() < edges:
        raise RuntimeError("the batch has too few edges")
    return off, *_thin(u, v, edges, gen)


def _ordered(case, n, u, v, gen):
    """Both directions of every edge in the case's order, int32."""
    src, dst = torch.cat([u, v]), torch.cat([v, u])
    if case["order"] == "rows":
        keys = torch.sort(src * n + dst).values
        src, dst = keys // n, keys % n
    elif case["order"] == "shuffled":
        at = torch.randperm(src.numel(), generator=gen, device="cuda")
        src, dst = src[at], dst[at]
    return src.int(), dst.int()


def _tsv(src, dst):
    """The text of 1-based "dst src 1" lines as bytes on the GPU."""
    columns, keep = [], []

    def text(c):
        columns.append(torch.full_like(dst, ord(c), dtype=torch.uint8))
        keep.append(torch.ones_like(dst, dtype=torch.bool))

    for ids, after in ((dst, "\t"), (src, "\t")):
        ids = ids.long() + 1
        for p in range(len(str(int(ids.max()))) - 1, -1, -1):
            columns.append((ids // 10**p % 10 + ord("0")).byte())
            keep.append(ids >= 10**p)
        text(after)
    text("1")
    text("\n")
    return torch.stack(columns, 1)[torch.stack(keep, 1)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    state = dict(op=op)
    if op == "batch":
        off, u, v = _batch(case, gen)
        n = off[-1]
        src, dst = _ordered(case, n, u, v, gen)
        state["offsets"] = torch.tensor(off, dtype=torch.int32, device="cuda")
        state["k_max"] = torch.zeros(case["graphs"], dtype=torch.int32, device="cuda")
    else:
        n = case["n"]
        src, dst = ([x.int() for x in _rmat(n, case["edges"], gen)] if op == "symmetrize"
                    else _ordered(case, n, *_simple(case, gen), gen))
    if op == "host":
        state["graph"] = kt.COOGraph(n, *(x.cpu().numpy().view(np.uint32) for x in (src, dst)))
        return state
    N = src.numel()
    state["engine"] = kt.Engine(0)
    if op == "parse":
        state.update(text=_tsv(src, dst), src=torch.zeros_like(src), dst=torch.zeros_like(dst))
    else:
        state["engine"].reserve(n, N)
        state.update(n=n, src=src.contiguous(), dst=dst.contiguous())
    if op in ("decompose", "batch"):
        state["truss"] = torch.zeros(N, dtype=torch.int32, device="cuda")
        state.setdefault("k_max", torch.zeros(1, dtype=torch.int32, device="cuda"))
    elif op == "ktruss":
        state.update(keep=torch.zeros(N, dtype=torch.uint8, device="cuda"), k=case["k"])
    elif op == "symmetrize":
        state["out"] = torch.zeros((2, 2 * N), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the engine has a stream of its own
    return state


def run(state):
    op = state["op"]
    if op == "host":
        truss, k_max = kt.decompose(state["graph"])
        return truss, k_max
    e, src, dst = state["engine"], state["src"], state["dst"]
    if op == "parse":
        text = state["text"]
        entries, n = e.parse_tsv(text.data_ptr(), text.numel(), src.data_ptr(), dst.data_ptr(), src.numel())
        return src, dst, entries, n
    if op == "symmetrize":
        out = state["out"]
        made = e.symmetrize(src.data_ptr(), dst.data_ptr(), src.numel(), state["n"], out[0].data_ptr(),
                            out[1].data_ptr(), out.shape[1])
        return out, made  # entries past the last one made stay zero
    if op == "ktruss":
        e.ktruss(src.data_ptr(), dst.data_ptr(), src.numel(), state["n"], state["k"], state["keep"].data_ptr())
        return state["keep"]
    truss, k_max = state["truss"], state["k_max"]
    if op == "decompose":
        e.decompose(src.data_ptr(), dst.data_ptr(), src.numel(), state["n"], truss.data_ptr(), k_max.data_ptr())
    else:
        e.decompose_batch(src.data_ptr(), dst.data_ptr(), src.numel(), state["n"], state["offsets"].data_ptr(),
                          k_max.numel(), truss.data_ptr(), k_max.data_ptr())
    return truss, k_max


def work(case):
    """Bytes of the inputs and outputs."""
    op = case["op"]
    if op == "batch":  # a graph has about 7 edges a vertex
        lo, hi = case["n_min"], case["n_max"]
        return dict(bytes=12 * 2 * 7 * case["graphs"] * (hi - lo) / math.log(hi / lo), flops=0)
    m = case["edges"]
    if op == "symmetrize":
        return dict(bytes=8 * m + 16 * m, flops=0)
    if op == "parse":  # two ids, a weight, separators; two words an entry
        return dict(bytes=2 * m * (2 * len(str(case["n"])) + 4) + 8 * 2 * m, flops=0)
    return dict(bytes=(8 + (1 if op == "ktruss" else 4)) * 2 * m, flops=0)
