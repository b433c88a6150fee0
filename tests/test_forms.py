"""The rules that choose a batch's form of stepping (csrc/bd_forms.h), on the
host against a model of the device: 148 SMs, two CTAs of a cluster kernel per
SM, one of the group kernel."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "bd-simulations_b200", "csrc")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "bd_forms.h"
using namespace bd;
// argv: piped, most runs, then N Z idgas of the kinds of run, taken in turn
int main(int argc, char** argv) {
  const bool piped = std::atoi(argv[1]) != 0;
  const int most = std::atoi(argv[2]);
  std::vector<FormRun> kinds;
  for (int a = 3; a + 2 < argc; a += 3) {
    FormRun r{};
    r.N = std::atoi(argv[a]), r.Z = std::atoi(argv[a + 1]), r.idgas = std::atoi(argv[a + 2]) != 0;
    kinds.push_back(r);
  }
  for (int n = 1; n <= most; n++) {
    std::vector<FormRun> runs;
    for (int k = 0; k < n; k++) runs.push_back(kinds[k % kinds.size()]);
    auto held = [&](size_t k, int cs) { return runs[k].Z > 1024 ? 0 : cs == 16 ? 16 : 296 / cs; };
    const BatchForm f = choose_batch_form(runs, held, n <= 148 ? 148 : 0, piped);
    double part = 0.0;
    long long ctas = 0;
    for (size_t k = 0; k < f.ctas.size(); k++) {
      if (f.ctas[k] < 1 || f.ctas[k] > 148) return 2;
      ctas += f.ctas[k];
      if (f.step == BATCH_CLUSTERS) {
        const int h = held(k, f.ctas[k]);
        if (h <= 0) return 3;
        part += 1.0 / h;
      }
    }
    std::printf("%d %d %zu %lld %.6f\n", n, (int)f.step, f.ctas.size(), ctas, part);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I" + CSRC, str(d / "h.cpp"), "-o", str(d / "h")],
                   check=True)
    return str(d / "h")


def _forms(harness, piped, most, kinds):
    o = subprocess.run([harness, str(piped), str(most)] + [str(v) for k in kinds for v in k], check=True,
                       capture_output=True, text=True).stdout
    return [[float(v) for v in line.split()] for line in o.splitlines()]


LAUNCHES, CLUSTERS, GROUPS = 0, 1, 2


@pytest.mark.parametrize("piped", [0, 1])
@pytest.mark.parametrize("kinds", [[(300, 24, 0)], [(20, 8, 0)], [(4000, 96, 0)], [(500, 64, 1)], [(100000, 768, 0)],
                                   [(50, 16, 0), (3000, 384, 0), (500, 64, 1)], [(900, 1024, 0)]])
def test_a_form_is_taken_only_where_it_fits(harness, piped, kinds):
    """1 to 1000 runs: clusters only when every run's are resident together,
    groups only with a CTA for every run and no more than there are, the
    launch-per-step form otherwise."""
    rows = _forms(harness, piped, 1000, kinds)
    assert len(rows) == 1000
    for n, step, given, ctas, part in rows:
        if step == LAUNCHES:
            assert given == 0
        else:
            assert given == n
        if step == CLUSTERS:
            assert part <= 1.0 + 1e-9
        if step == GROUPS:
            assert n <= 148 and ctas <= 148
        if n > 296:
            assert step == LAUNCHES


def test_small_batches_take_one_launch_for_many_steps(harness):
    assert all(r[1] != LAUNCHES for r in _forms(harness, 0, 290, [(300, 24, 0)]))
    assert all(r[1] != LAUNCHES for r in _forms(harness, 1, 8, [(2000, 64, 0)]))


def test_runs_no_cluster_holds_take_launches(harness):
    assert all(r[1] == LAUNCHES for r in _forms(harness, 0, 400, [(1000, 1152, 0)]) if r[0] > 148)
