"""A device wait that gives up in any form of stepping (one-step launch,
resident grid, groups of CTAs, cooperative tail): whatever the caller does
next, nothing moves or sorts the run before the synchronising call that
reports BD_ERR_TIMEOUT and puts it back, and it steps on with the bits of a
run that never failed. The hook makes one CTA leave instead of arriving and
lowers the poll limit (no fault, no endless wait)."""
import numpy as np
import pytest

from test_gpu_resident import _lattice, _params, _same

pytestmark = pytest.mark.gpu

BD_ERR_STATE, BD_ERR_TIMEOUT = -5, -10


def _timeout(gpu, fn, *a):
    with pytest.raises(gpu.BdError) as e:
        fn(*a)
    assert e.value.status == BD_ERR_TIMEOUT


def _pair(gpu, p, seed=4):
    start = _lattice(p, 9)
    a, b = gpu.Run(p, seed=seed), gpu.Run(p, seed=seed)
    for r in (a, b):
        r.set_positions_all(start)
        r.zeitschritte(3)
    return a, b


# a cluster, the resident grid, a launch per step, and runs that step pipelined
# when asked for eight steps or more
FORMS = [(400, 301, 32), (3000, 2001, 128), (3000, 2001, 1024), (65536, 65536, 512), (150000, 120000, 256)]


@pytest.mark.parametrize("barrier", [1, 2, 3])
@pytest.mark.parametrize("n1,n2,mesh", FORMS)
def test_failed_single_step_then_a_call_of_many(gpu, n1, n2, mesh, barrier):
    a, b = _pair(gpu, _params(gpu, n1, n2, mesh, False))
    a._call("bd_inject_barrier_timeout", barrier, 2000)
    a.zeitschritt()  # queued: its wait gives up on the device
    _timeout(gpu, a.zeitschritte, 20)
    assert a.step_count() == 3 and a.time() == b.time()
    _same(a.get_positions(), b.get_positions())
    for r in (a, b):
        r.zeitschritte(20)
        r.zeitschritt()
        r.sync()
    _same(a.get_positions(), b.get_positions())
    assert a.step_count() == b.step_count() == 24 and a.time() == b.time()


@pytest.mark.parametrize("n1,n2,mesh", FORMS)
def test_failed_step_inside_a_call(gpu, n1, n2, mesh):
    """The second barrier of the fourth step of one resident launch."""
    a, b = _pair(gpu, _params(gpu, n1, n2, mesh, False))
    a._call("bd_inject_wait_timeout", 4 * 3 + 2, 20000)
    _timeout(gpu, a.zeitschritte, 10)
    assert a.step_count() == 6
    b.zeitschritte(3)
    _same(a.get_positions(), b.get_positions())
    for r in (a, b):
        r.zeitschritte(9)
    _same(a.get_positions(), b.get_positions())
    assert a.time() == b.time()


@pytest.mark.parametrize("call", ["set_positions", "refresh", "debug", "stage"])
def test_failed_step_then_sorting_calls(gpu, call):
    """Calls that count and sort particles of their own: not on top of the
    counts the failed step left."""
    p = _params(gpu, 3000, 2001, 128, False)
    a, b = _pair(gpu, p)
    a._call("bd_inject_barrier_timeout", 2, 2000)
    a.zeitschritt()
    if call == "set_positions":
        a.set_positions_all(_lattice(p, 77))
        _timeout(gpu, a.sync)
    elif call == "refresh":
        _timeout(gpu, a.refresh_erwNachbar)
    elif call == "debug":
        _timeout(gpu, a.zeitschritt_debug, 0.05)
    else:
        a.stage_times(2)
        _timeout(gpu, a.sync)
    assert a.step_count() == 3
    _same(a.get_positions(), b.get_positions())
    for r in (a, b):
        r.zeitschritte(5)
    _same(a.get_positions(), b.get_positions())


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("barrier", [1, 2, 3])
def test_group_of_a_batch_fails(gpu, adaptive, barrier):
    """One run's group gives up; the next calls take the group form and the
    launch-per-step form; the other runs step on."""
    sizes = [(60, 41, 16), (3000, 2501, 384), (500, 400, 64), (9000, 8000, 256)]
    runs = [_params(gpu, n1, n2, m, adaptive and k != 3, scheme=2) for k, (n1, n2, m) in enumerate(sizes)]
    a, b = gpu.Batch(runs, [3, 4, 5, 6]), gpu.Batch(runs, [3, 4, 5, 6])
    for x in (a, b):
        for k, p in enumerate(runs):
            x.set_positions(k, _lattice(p, 70 + k))
    lib = gpu.lib()
    assert lib.bd_batch_inject_wait_timeout(a.h, 4, 1, 100) == -1
    assert lib.bd_batch_inject_wait_timeout(a.h, 1, 0, 100) == -1
    assert lib.bd_batch_inject_wait_timeout(a.h, 1, barrier, 20000) == 0
    a.step(5)
    a.step(1)
    a.step(2)
    _timeout(gpu, a.sync)
    before = a.get_positions(1)
    assert a.time(1) == 0.0
    _same(before, b.get_positions(1))
    b.step(8)
    for k in (0, 2, 3):
        _same(a.get_positions(k), b.get_positions(k))
        assert a.time(k) == b.time(k)
    a.step(8)
    a.sync()
    _same(a.get_positions(1), b.get_positions(1))
    b.step(8)
    for k in (0, 2, 3):
        _same(a.get_positions(k), b.get_positions(k))


def test_cooperative_tail_fails(gpu):
    """Step form 1: a failed wait concerns every run of the batch, also when
    the form is changed before the failure is reported."""
    runs = [_params(gpu, n1, n2, m, False) for n1, n2, m in ((300, 201, 32), (900, 800, 64), (2000, 1500, 128))]
    a, b = gpu.Batch(runs, [1, 2, 3]), gpu.Batch(runs, [1, 2, 3])
    for x in (a, b):
        for k, p in enumerate(runs):
            x.set_positions(k, _lattice(p, 50 + k))
        x.set_step_form(1, 4)
        x.step(2)
        x.sync()
    assert a.launches_per_step() == 2
    assert gpu.lib().bd_batch_inject_wait_timeout(a.h, 0, 1, 2000) == 0
    a.step(3)
    a.set_step_form(0)
    a.step(1)
    a.step(4)
    _timeout(gpu, a.sync)
    for x in (a, b):
        x.set_step_form(0)
    for k in range(3):
        _same(a.get_positions(k), b.get_positions(k))
        assert a.time(k) == b.time(k)
    for x in (a, b):
        x.step(6)
    for k in range(3):
        _same(a.get_positions(k), b.get_positions(k))


def test_wait_hook_refused_without_grid_barriers(gpu):
    p = _params(gpu, 1000, 901, 1152, True)  # beyond the resident step: stage kernels
    r = gpu.Run(p, seed=1)
    r.set_positions_all(_lattice(p, 1))
    for args, status in (((1, 100), BD_ERR_STATE), ((0, 100), -1), ((1, 0), -1)):
        with pytest.raises(gpu.BdError) as e:
            r._call("bd_inject_wait_timeout", *args)
        assert e.value.status == status


# a group barrier behind each phase of an adaptive step, the dt bound's
# (2) among them; a mesh of each class, 2^k and 3 * 2^k and other factors of 3
@pytest.mark.parametrize("barrier", [1, 2, 3, 4])
@pytest.mark.parametrize("n1,n2,mesh", [(400, 301, 64), (900, 800, 144), (2000, 1501, 384)])
def test_adaptive_step_reports_its_failed_wait(gpu, n1, n2, mesh, barrier):
    p = _params(gpu, n1, n2, mesh, True, obs_dt=0.01)
    start = _lattice(p, 9)
    a, b = gpu.Run(p, seed=4), gpu.Run(p, seed=4)
    for r in (a, b):
        r.set_positions_all(start)
    # the run's first step: no step length to repeat
    a._call("bd_inject_wait_timeout", barrier, 20000)
    _timeout(gpu, a.zeitschritte_bis_obs)
    assert a.step_count() == 0 and a.time() == 0.0
    _same(a.get_positions(), b.get_positions())
    assert a.zeitschritt() == b.zeitschritt()
    a._call("bd_inject_wait_timeout", barrier, 20000)
    _timeout(gpu, a.zeitschritt)
    assert a.step_count() == 1 and a.time() == b.time()
    _same(a.get_positions(), b.get_positions())
    # the failed steps added nothing to the time since the observation
    assert a.zeitschritte_bis_obs() == b.zeitschritte_bis_obs()
    _same(a.get_positions(), b.get_positions())
    fa, fb = a.get_forces(), b.get_forces()
    for k in fa:
        assert np.array_equal(fa[k], fb[k])
    assert a.time() == b.time()
