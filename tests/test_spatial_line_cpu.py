"""The lines from which a whole run sorts its points (csrc/host/spatial_line.hpp)
against measured loops, plain and sorted: the side that they choose."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "cl-kmeans_gb300", "csrc", "host", "spatial_line.hpp")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include HEADER
int main() {
    char strategy[32];
    unsigned long long n;
    unsigned k, iterations;
    while (scanf("%31s %llu %u %u", strategy, &n, &k, &iterations) == 4)
        printf("%d\n", (int)(strcmp(strategy, "single_stage") == 0
                                  ? Clustering::single_stage_spatial_pays(n, k, iterations)
                                  : Clustering::three_stage_spatial_pays(n, k, iterations)));
}
"""

# n, k, us of a loop of 8 iterations plain and sorted, of 30 plain and sorted (d = 4, blobs)
LOOPS = {
    "single_stage": [
        (1 << 20, 4, 120, 190, 424, 429), (1 << 20, 10, 139, 215, 500, 531), (1 << 20, 20, 194, 249, 688, 653),
        (1 << 20, 32, 229, 267, 814, 715), (1 << 22, 4, 190, 347, 686, 810), (1 << 22, 10, 257, 365, 936, 858),
        (1 << 22, 20, 403, 442, 1481, 1116), (1 << 22, 32, 556, 481, 2046, 1227), (1 << 24, 4, 557, 959, 2047, 2257),
        (1 << 24, 10, 771, 990, 2842, 2352), (1 << 24, 20, 1351, 1314, 5024, 3413),
        (1 << 24, 32, 1786, 1384, 6655, 3545),
    ],
    "three_stage": [
        (1 << 20, 4, 244, 303, 882, 848), (1 << 20, 10, 344, 335, 1259, 945), (1 << 20, 20, 365, 369, 1337, 1076),
        (1 << 20, 32, 406, 396, 1485, 1179), (1 << 22, 4, 377, 542, 1368, 1556), (1 << 22, 10, 519, 580, 1895, 1627),
        (1 << 22, 20, 647, 651, 2370, 1866), (1 << 22, 32, 773, 684, 2841, 1952),
        (1 << 24, 4, 1186, 1634, 4369, 4797), (1 << 24, 10, 1420, 1730, 5264, 5130),
        (1 << 24, 20, 1952, 1933, 7249, 5743), (1 << 24, 32, 2390, 1977, 8918, 5734),
    ],
}
# single loops: n, d, k, iterations, us plain, us sorted
SINGLE = {
    "single_stage": [(1 << 20, 4, 10, 8, 138, 216), (1 << 20, 4, 10, 30, 500, 532), (1 << 23, 4, 10, 30, 1623, 1464),
                     (1 << 23, 8, 30, 8, 1631, 1469), (1 << 23, 4, 32, 15, 1814, 1237), (1 << 23, 8, 8, 15, 1152, 1494)],
    "three_stage": [(1 << 20, 4, 10, 15, 629, 536), (1 << 23, 4, 10, 15, 1568, 1659), (1 << 23, 8, 30, 8, 2056, 1892)],
}


@pytest.fixture(scope="module")
def pays(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not installed")
    d = tmp_path_factory.mktemp("line")
    src, exe = d / "line.cpp", d / "line"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", '-DHEADER="%s"' % HEADER, str(src), "-o", str(exe)], check=True)

    def ask(queries):
        text = "\n".join("%s %d %d %d" % q for q in queries)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
        assert len(out) == len(queries)
        return [o == "1" for o in out]
    return ask


def test_measured_loops_take_the_faster_side(pays):
    cases = [(s,) + c for s, cs in SINGLE.items() for c in cs]
    for c, sorts in zip(cases, pays([(s, n, k, it) for s, n, _, k, it, _, _ in cases])):
        assert sorts == (c[6] < c[5]), c


def test_no_loop_loses_much(pays):
    queries, times = [], []
    for s, loops in LOOPS.items():
        for n, k, p8, s8, p30, s30 in loops:
            for it in (8, 10, 12, 15, 20, 25, 30, 40, 50):
                queries.append((s, n, k, it))
                times.append((p8 + (it - 8) * (p30 - p8) / 22, s8 + (it - 8) * (s30 - s8) / 22))
    loss = []
    for q, (plain, by_order), sorts in zip(queries, times, pays(queries)):
        loss.append((by_order if sorts else plain) / min(plain, by_order) - 1)
        assert loss[-1] <= 0.12, (q, plain, by_order)
    assert sum(loss) / len(loss) <= 0.01
