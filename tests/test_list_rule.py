"""The rules of the triangle lists (csrc/kt_list_rule.h), built for the host: the buffer for uncounted graphs
covers every graph of that many edges, a repeated call whose buffer was lost or shrank walks rows instead of
writing to it, buffers keep to their limit, and which graphs walk."""
import math
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("rule") / "list_rule_driver")
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "ktruss-explorer_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "compat", "list_rule_driver.cpp")], check=True)

    def run(*queries):
        text = "".join(" ".join(map(str, q)) + "\n" for q in queries)
        r = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
        return [int(x) for x in r.stdout.split()]

    return run


def _most_triangles(m):
    """Kruskal-Katona: the clique of c vertices that m edges hold, and one more vertex for the rest."""
    c = (1 + math.isqrt(1 + 8 * m)) // 2
    rest = m - math.comb(c, 2)
    return math.comb(c, 3) + math.comb(rest, 2)


def test_uncounted_lists_fit_every_graph(ask):
    sizes = list(range(1, 2000)) + [4950, 5049, 32385, 32766, 32767, 32768, 1 << 20, 123456789, (1 << 31) - 1]
    for m, most in zip(sizes, ask(*[("most", m) for m in sizes])):
        assert most >= 3 * _most_triangles(m), m
    cap, = ask(("most", 1 << 15))
    assert cap * 8 < 68e6
    assert ask(("small", 1 << 15, cap), ("small", 1 << 15, cap - 1), ("small", (1 << 15) + 1, 1 << 62),
               ("small", 1, 0)) == [1, 0, 0, 0]


def test_a_repeated_call_without_its_buffer_walks(ask):
    # the buffer it had, a larger one, a smaller one, none; a call that walked
    assert ask(("repeat", 100, 100), ("repeat", 100, 101), ("repeat", 100, 99), ("repeat", 1, 0), ("repeat", 0, 0),
               ("repeat", 0, 100)) == [1, 1, 0, 0, 0, 0]


def test_buffers_keep_to_the_limit(ask):
    none = (1 << 64) - 1
    cases = [(0, none, 1), (0, 8, 1), (0, 7, 0), (0, 0, 0), (15, none, 15), (16, none, 17), (16, 17 * 8, 17),
             (16, 17 * 8 - 1, 16), (16, 16 * 8, 16), (16, 16 * 8 - 1, 0), (5 << 30, none, (5 << 30) + (5 << 26))]
    assert ask(*[("buffer", t, limit) for t, limit, _ in cases]) == [want for *_, want in cases]


def _cliques(size, count):
    m = count * math.comb(size, 2)
    return m, (size - 2) * m


def test_which_graphs_walk(ask):
    def walks(*graphs):  # (edges, list entries, near-cliques' entries, least support[, edges in triangles])
        return ask(*[("walks", g[0], g[4] if len(g) > 4 else g[0], *g[1:4]) for g in graphs])

    near = [(c, (*_cliques(*c), _cliques(*c)[1], 0), walk) for c, walk in [
        ((500, 2), 1), ((400, 1), 1), ((200, 6), 1), ((100, 26), 0), ((60, 140), 0), ((60, 160), 1), ((20, 1500), 0),
        ((514, 3), 1), ((516, 1), 1)]]
    for (c, _, walk), got in zip(near, walks(*[g for _, g, _ in near])):
        assert got == walk, c
    total = 1 << 25
    assert walks((200000, total, total, 0), (200000, total, total - total // 256, 0),
                 (200000, total, total - total // 256 - 1, 0), (200000, 1 << 24, 1 << 24, 0),
                 (200000, (1 << 24) - 1, (1 << 24) - 1, 0), (1 << 18, 1 << 23, 1 << 23, 0),
                 (1 << 18, (1 << 23) - 1, (1 << 23) - 1, 0), (1 << 18, 1 << 24, 3 << 22, 0),
                 (1 << 18, 1 << 24, (3 << 22) + 1, 0)) == [1, 1, 0, 1, 0, 1, 0, 0, 1]
    # density; dense and even
    m = 50000
    assert walks((m, 512 * m + 511, 0, 0), (m, 512 * (m + 1), 0, 0), (40000, 0, 0, 0, 0),
                 (1 << 18, (512 << 18) + 511, 0, 400), (1 << 18, 512 * ((1 << 18) + 1), 0, 0),
                 (m, 400 * m, 0, 320), (m, 400 * m, 0, 319), (m, 320 * m, 0, 320),
                 (m, 320 * (m + 1), 0, 260), (m, 320 * (m + 1), 0, 250),
                 (1 << 18, 400 << 18, 0, 400)) == [0, 1, 0, 0, 1, 1, 0, 0, 1, 0, 0]
    # edges in no triangle do not thin an even graph out
    assert walks((10 * m, 512 * m + 511, 0, 512, m), (10 * m, 512 * (m + 1), 0, 350, m),
                 (10 * m, 512 * (m + 1), 0, 341, m), (200000, 400 * m, 0, 320, m), (200000, 400 * m, 0, 319, m),
                 (10 * m, 400 * m, 0, 400, m), (10 * m, 512 * 10 * m + 511, 0, 0, m),
                 (10 * m, 512 * (10 * m + 1), 0, 0, m)) == [0, 1, 0, 1, 0, 0, 0, 1]
