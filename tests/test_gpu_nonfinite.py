"""Positions that leave the finite range: a step length of 1e30 throws every
particle, at T = 1 to finite offsets far beyond what re-binning reaches, at
T = 1e30 to infinity. Every form of stepping indexes the mesh within its
arrays, reports BD_ERR_NONFINITE and leaves the device usable."""
import numpy as np
import pytest

from test_gpu_resident import _lattice, _params, _same

pytestmark = pytest.mark.gpu

BD_ERR_NONFINITE, BD_ERR_TIMEOUT = -8, -10


def _status(gpu, fn, *a):
    try:
        fn(*a)
    except gpu.BdError as e:
        return e.status
    return 0


def _thrown(gpu, n1, n2, mesh, T, scheme=2):
    return dict(_params(gpu, n1, n2, mesh, False, scheme=scheme), dt_max=1e30, T=T)


@pytest.mark.parametrize("T", [1.0, 1e30])
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("mesh", [8, 64, 96, 144, 1024, 2048])
def test_thrown_particles(gpu, mesh, scheme, T):
    p = _thrown(gpu, 700, 601, mesh, T, scheme)
    r = gpu.Run(p, seed=2)
    r.set_positions_all(_lattice(p, 3))
    got = [_status(gpu, f, n) for f, n in ((r.zeitschritte, 1), (r.zeitschritte, 3), (r.zeitschritte, 9))]
    assert all(s in (0, BD_ERR_NONFINITE) for s in got)
    if T > 1:
        assert got == [BD_ERR_NONFINITE] * 3
    r.stage_times(2)
    cells = np.concatenate([q[0] for q in r.get_positions().values()])
    assert cells.min() >= 0 and cells.max() < int(p["L"] / 2 ** (1 / 6))
    r.close()
    # the device steps on
    q = _params(gpu, 300, 201, 32, False)
    a, b = gpu.Run(q, seed=1), gpu.Run(q, seed=1)
    for x in (a, b):
        x.set_positions_all(_lattice(q, 1))
    a.zeitschritte(3)
    b.stage_times(3)
    _same(a.get_positions(), b.get_positions())


@pytest.mark.parametrize("meshes", [(64, 128, 32), (64, 96, 144), (96, 384, 16)])
def test_thrown_run_of_a_batch(gpu, meshes):
    """One run of a batch is thrown, the others step with their own bits."""
    runs = [_params(gpu, 700, 501, m, False) for m in meshes]
    runs[1] = _thrown(gpu, 700, 501, meshes[1], 1e30)
    seeds = [1, 2, 3]
    b = gpu.Batch(runs, seeds)
    for k, p in enumerate(runs):
        b.set_positions(k, _lattice(p, 20 + k))
    for n in (4, 1):
        b.step(n)
        assert _status(gpu, b.sync) == BD_ERR_NONFINITE
    for k in (0, 2):
        r = gpu.Run(runs[k], seed=seeds[k])
        r.set_positions_all(_lattice(runs[k], 20 + k))
        r.stage_times(5)
        _same(b.get_positions(k), r.get_positions())


def test_thrown_run_does_not_hide_another_runs_failed_wait(gpu):
    """Both errors in one batch: the run whose wait gave up is put back and
    reported, the thrown one's error stays."""
    meshes = (96, 384, 64)
    runs = [_params(gpu, 900, 601, m, k == 1) for k, m in enumerate(meshes)]
    runs[0] = _thrown(gpu, 900, 601, meshes[0], 1e30)
    b = gpu.Batch(runs, [1, 2, 3])
    for k, p in enumerate(runs):
        b.set_positions(k, _lattice(p, 30 + k))
    assert gpu.lib().bd_batch_inject_wait_timeout(b.h, 1, 3, 20000) == 0
    b.step(2)
    assert _status(gpu, b.sync) == BD_ERR_TIMEOUT
    assert _status(gpu, b.sync) == BD_ERR_NONFINITE
    assert b.time(1) == 0.0
    b.step(4)
    assert _status(gpu, b.sync) == BD_ERR_NONFINITE
    for k, n in ((1, 4), (2, 6)):
        r = gpu.Run(runs[k], seed=k + 1)
        r.set_positions_all(_lattice(runs[k], 30 + k))
        r.stage_times(n)
        _same(b.get_positions(k), r.get_positions())
        assert b.time(k) == r.time()
