"""The form that a batch's steps take follows estimates of all three forms: a
resident form only where it is expected to be faster than launches. Batches
measured in each form on a B200."""
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
// argv: piped, runs, then N Z idgas adaptive of the kinds of run, taken in turn
int main(int argc, char** argv) {
  const int n = std::atoi(argv[2]);
  std::vector<FormRun> kinds, runs;
  for (int a = 3; a + 3 < argc; a += 4)
    kinds.push_back({std::atoi(argv[a]), std::atoi(argv[a + 1]), std::atoi(argv[a + 2]) != 0, std::atoi(argv[a + 3]) != 0});
  for (int k = 0; k < n; k++) runs.push_back(kinds[k % kinds.size()]);
  auto held = [&](size_t k, int cs) { return runs[k].Z > 1024 ? 0 : cs == 16 ? 8 : 296 / cs; };
  const BatchForm f = choose_batch_form(runs, held, n <= 148 ? 148 : 0, std::atoi(argv[1]) != 0, 148);
  std::printf("%d %.3f %d %d %d\n", (int)f.step, f.us, idgas_stage_kernels(kinds[0].N, kinds[0].Z),
              steps_per_launch(f.us), steps_per_launch(estimate_single(kinds[0])));
  return 0;
}
"""

LAUNCHES, CLUSTERS, GROUPS = 0, 1, 2


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("estimates")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I" + CSRC, str(d / "h.cpp"), "-o", str(d / "h")],
                   check=True)
    return str(d / "h")


def _form(harness, piped, runs, kinds):
    o = subprocess.run([harness, str(piped), str(runs)] + [str(v) for k in kinds for v in k], check=True,
                       capture_output=True, text=True).stdout.split()
    return int(o[0]), float(o[1]), int(o[2]), int(o[3]), int(o[4])


# us per step measured in launches, on clusters, in groups (None: do not fit)
@pytest.mark.parametrize("piped,runs,kinds,us", [
    (0, 256, [(826, z, 0, 1) for z in (32, 64, 128, 256, 512, 1024)], (1464, 6580, None)),
    (0, 200, [(4000, 256, 0, 1)], (411, 721, None)),
    (0, 148, [(4000, 256, 0, 1)], (297, 612, 453)),
    (0, 200, [(1337, z, 0, 1) for z in (48, 96, 192, 384, 768)], (1752, 3458, None)),
    (1, 2, [(54436, 256, 0, 0)], (31.0, 84, 31.5)),
    (1, 71, [(2325, 1024, 0, 0)], (1567, 2416, 3184)),
    (0, 169, [(300, 288, 1, 0), (2000, 288, 1, 0), (90000, 288, 1, 0)], (286, 445, None)),
    (0, 290, [(479, 32, 0, 1)], (57, 32, None)),
    (0, 256, [(16000, 192, 0, 1)], (1191, 830, None)),
    (0, 16, [(1000, 128, 0, 1)], (50.7, 23.3, 23.5)),
    (0, 120, [(1164, 384, 0, 1)], (1042, 599, 774)),
    (1, 4, [(795, 32, 0, 0)], (20, 11, 16)),
    (0, 2, [(988, 768, 0, 1)], (113, 204, 70)),
    (0, 256, [(305, 32, 1, 0)], (16.2, 11.5, None)),
])
def test_the_fastest_form(harness, piped, runs, kinds, us):
    form, estimate = _form(harness, piped, runs, kinds)[:2]
    best = min((t, k) for k, t in enumerate(us) if t is not None)[1]
    assert form == best or us[form] < 1.1 * us[best]
    if not piped:  # the pipelined step's estimate counts particles only
        assert 0.5 * us[form] < estimate < 2.0 * us[form]


@pytest.mark.parametrize("n,steps,launches", [(6000, 1, 0), (6001, 1, 1), (6001, 2, 0), (65536, 400, 0), (65537, 400, 1)])
def test_single_ideal_gas_runs(harness, n, steps, launches):
    assert _form(harness, 0, 1, [(n, steps, 1, 0)])[2] == launches


# us per step measured: batches, single runs
@pytest.mark.parametrize("runs,kind,us", [(256, (1000, 768, 0, 1), 5368), (148, (1000, 768, 0, 0), 3326),
                                          (256, (16000, 192, 0, 1), 830), (290, (479, 32, 0, 1), 32),
                                          (1, (2000, 128, 0, 0), 15), (1, (64000, 648, 0, 1), 78),
                                          (1, (262144, 1024, 0, 1), 83), (1, (3000000, 1024, 0, 1), 591)])
def test_a_launch_takes_about_50_ms_at_most(harness, runs, kind, us):
    f = _form(harness, 0, runs, [kind])
    steps = f[4] if runs == 1 else f[3]
    assert runs == 1 or f[0] != LAUNCHES
    assert 1 <= steps <= 1024 and steps * us <= 100e3
    assert steps == 1024 or steps * us >= 25e3
