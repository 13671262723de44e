"""The host rules of the triangle lists' buffer (csrc/kt_list_rule.h), built for the host: its size for
uncounted graphs covers every graph of that many edges, and a repeated call whose buffer was lost or shrank
walks rows instead of writing to it."""
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
