"""The CTAs that a work slot gets, compiled for the host (148 SMs, every cluster fits)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include <cstdlib>
#include "team_rule.cuh"
int main(int, char** a) {
  const int n = atoi(a[1]), slots = atoi(a[2]);
  auto fit = [](int c) { return 148 / c; };
  std::printf("%d %d", negf::team_rule(n, slots, 148, fit), negf::team_rule(negf::ls_team_n(n), slots, 148, fit));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "r.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "dpnegf_b200", "csrc"), "r.cpp", "-o", "r"], cwd=d,
                   check=True)
    return lambda n, slots: tuple(map(int, subprocess.run([str(d / "r"), str(n), str(slots)], check=True,
                                                          capture_output=True, text=True).stdout.split()))


@pytest.mark.parametrize("n", [1, 16, 17, 24, 32, 33, 48])
@pytest.mark.parametrize("slots", [1, 18, 74, 148])
def test_small_leads_stay_on_one_cta(rule, n, slots):
    assert rule(n, slots)[1] == 1


@pytest.mark.parametrize("n,slots,sweep,lead", [(32, 1, 1, 1), (33, 1, 2, 1), (49, 1, 2, 8), (64, 18, 2, 8), (65, 18, 4, 8),
                                                (96, 37, 4, 4), (128, 18, 8, 8), (128, 19, 4, 4), (128, 74, 2, 2),
                                                (128, 75, 1, 1), (512, 148, 1, 1)])
def test_clusters_by_size_and_slots(rule, n, slots, sweep, lead):
    assert rule(n, slots) == (sweep, lead)
