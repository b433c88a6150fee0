"""A program that resets the device between its contexts (in a process of its
own here) can go on: what a kernel needs set is set for each engine."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, "tests")
import conftest
import bdsim as gpu
from test_gpu_resident import _lattice, _params

def use():
    # the resident grid, one cluster, the one-step launch; a batch on clusters,
    # one whose runs share a cooperative grid
    out = []
    for n, mesh in ((3000, 384), (1000, 128), (3000, 512)):
        p = _params(gpu, n, n, mesh, False)
        r = gpu.Run(p, seed=1)
        r.set_positions_all(_lattice(p, 2))
        r.zeitschritte(9)
        r.zeitschritt()
        r.sync()
        out.append(r.get_positions())
        r.close()
    for meshes in ((48, 48, 96), (384, 48)):
        ps = [_params(gpu, 900, 800, m, True) for m in meshes]
        b = gpu.Batch(ps, list(range(len(ps))))
        for k, p in enumerate(ps):
            b.set_positions(k, _lattice(p, k))
        b.step(6)
        b.sync()
        out += [b.get_positions(k) for k in range(len(ps))]
        b.close()
    return out

a = use()
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0
b = use()
for x, y in zip(a, b):
    for s in (0, 1):
        assert np.array_equal(x[s][0], y[s][0]) and np.array_equal(x[s][1], y[s][1])
print("same")
"""


def test_contexts_either_side_of_a_device_reset(gpu):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
