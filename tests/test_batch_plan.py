"""The hand-out of a batch's systems to teams of CTAs, on the host (csrc/batch_plan.h).

152 SMs take three CTAs each.  Where two an SM need as many rounds of teams as
three, three made uniform batches up to 1.4 times as slow as one CTA a system.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matrix-toolkits-java_gb300", "csrc")

PROGRAM = """
#include <cstdio>
#include <numeric>
#include "batch_plan.h"
int main(int argc, char **argv)
{
    std::vector<int> rows{0}, order;
    int n;
    while (std::scanf("%d", &n) == 1) rows.push_back(rows.back() + n);
    order.resize(rows.size() - 1);
    std::iota(order.begin(), order.end(), 0);
    int counts[mtjg::kTeamSizes];
    mtjg::batch_teams(rows.data(), order, counts);
    int at = 0;
    for (int c = 0; c < mtjg::kTeamSizes; at += counts[c++])
        std::printf("%d %d\\n", counts[c],
                    counts[c] ? mtjg::batch_per_sm(rows.data(), order.data() + at, counts[c], 8 >> c, 152) : 0);
    for (int s : order) std::printf("%d ", s);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(d / "t"), str(d / "t.cpp")], check=True)

    def run(sizes):
        out = subprocess.run([str(d / "t")], input=" ".join(map(str, sizes)), check=True, capture_output=True, text=True)
        lines = out.stdout.split("\n")
        return [tuple(map(int, l.split())) for l in lines[:4]], list(map(int, lines[4].split()))

    return run


def test_teams_by_rows(plan):
    sizes = [4095, 16384, 4096, 8191, 50000, 8192, 1, 0, 16383]
    per, order = plan(sizes)
    assert [c for c, _ in per] == [2, 2, 2, 3]
    assert order == [1, 4, 5, 8, 2, 3, 0, 6, 7]  # largest teams first, each in the order given


@pytest.mark.parametrize("count,rows,ctas", [
    (152, 6000, 3), (153, 6000, 3), (228, 6000, 3),  # one round by three
    (229, 6000, 2), (300, 6000, 2), (304, 6000, 2),  # two rounds either way
    (305, 6000, 3), (1200, 6000, 3),                 # more rounds by two
    (300, 8300, 3), (120, 8300, 2), (60, 20000, 2), (300, 17000, 3), (600, 1500, 3)])
def test_ctas_per_sm(plan, count, rows, ctas):
    per, _ = plan([rows] * count)
    assert [p for c, p in per if c] == [ctas]


def test_uneven_systems_keep_three(plan):
    """Longest first: the rounds overlap, and two an SM would only take longer."""
    per, _ = plan(sorted((16384 + 160 * k for k in range(200)), reverse=True))
    assert per[0] == (200, 3)
