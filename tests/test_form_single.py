"""The forms that a single run's calls of several steps take (csrc/bd_forms.h),
on either side of the sizes where they change."""
import subprocess

import pytest

from test_form_estimates import CSRC

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "bd_forms.h"
using namespace bd;
int main(int, char** argv) {
  const int N = std::atoi(argv[1]), Z = std::atoi(argv[2]), runs = std::atoi(argv[3]);
  std::printf("%d %d %d\n", pipelined_single(N, Z), launch_per_step_single(N, Z),
              step_kernel_prefetches((N + 255) / 256 * runs, runs, (double)N * runs, (double)Z * Z * runs));
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("single")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I" + CSRC, str(d / "h.cpp"), "-o", str(d / "h")],
                   check=True)
    return str(d / "h")


# particles, mesh, runs; pipelined, a launch per step otherwise, prefetching
# particle kernel
@pytest.mark.parametrize("n,mesh,runs,want", [
    (131071, 512, 1, (0, 0, 1)), (131072, 512, 1, (1, 0, 1)), (130816, 512, 1, (0, 0, 0)),
    (262143, 256, 1, (0, 0, 1)), (262144, 256, 1, (1, 0, 1)),
    (65536, 1024, 1, (0, 1, 0)), (131072, 1024, 1, (1, 1, 1)),
    # many particles to a mesh point
    (3000000, 256, 1, (1, 1, 0)), (3145728, 256, 1, (1, 1, 0)), (3145729, 256, 1, (0, 1, 0)),
    (1000000, 64, 1, (0, 1, 0)), (131072, 64, 1, (0, 1, 0)), (98304, 64, 1, (0, 0, 0)), (98305, 64, 1, (0, 1, 0)),
    (64000, 16, 1, (0, 1, 0)), (49999, 16, 1, (0, 0, 0)),
    # beyond the resident step's meshes
    (2000, 2048, 1, (1, 0, 0)), (4000000, 2048, 1, (1, 0, 1)), (262143, 4096, 1, (1, 0, 1)), (262144, 4096, 1, (0, 0, 1)),
    # batches
    (250000, 512, 8, (1, 0, 1)), (24000, 256, 256, (0, 0, 0)), (500000, 64, 2, (0, 1, 0)),
])
def test_single_run_rules(harness, n, mesh, runs, want):
    o = subprocess.run([harness, str(n), str(mesh), str(runs)], check=True, capture_output=True, text=True).stdout
    assert tuple(int(v) for v in o.split()) == want
