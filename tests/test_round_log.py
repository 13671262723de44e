"""The check of a decomposition's round log (round_follows, csrc/kt_device.cuh), built for the host: logs as the
oracle's rounds give them pass, and logs that no decomposition leaves behind do not."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def follows(tmp_path_factory):
    if not shutil.which("nvcc"):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("log") / "round_log_driver")
    r = subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "ktruss-explorer_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), "-o", exe,
                        os.path.join(ROOT, "tests", "compat", "round_log_driver.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def ask(rows):
        text = "".join(" ".join(map(str, r)) + "\n" for r in rows)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return [int(x) for x in out.split()]

    return ask


def _rows(log, m, k_max):
    """A log of (level, edges removed) as the arguments of its checks."""
    rows, before = [], 2
    for k, size in log:
        rows.append((k, before, k_max, size, m))
        m, before = m - size, k
    return rows


def test_logs_of_decompositions(follows):
    logs = [([(3, 5), (4, 2), (4, 1), (7, 9)], 17, 6), ([(3, 1)], 1, 2), ([(306, 4), (307, 2)], 6, 306),
            ([(5, 1), (5, 1), (5, 4294967293)], 4294967295, 4)]
    for log, m, k_max in logs:
        assert follows(_rows(log, m, k_max)) == [1] * len(log)


def test_inconsistent_logs(follows):
    assert follows([(2, 2, 6, 1, 9),    # a level below 3
                    (4, 5, 6, 1, 9),    # levels go down
                    (8, 5, 6, 1, 9),    # past the last level
                    (4, 4, 6, 0, 9),    # a round that removes nothing
                    (4, 4, 6, 10, 9),   # more than there is
                    (4, 4, 6, 1, 0)]) == [0] * 6
