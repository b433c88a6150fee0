"""What a program waits for the first time it makes a call: nothing that the
run's or the batch's creation could have done."""
import time

import pytest

from test_gpu_resident import _lattice, _params

pytestmark = pytest.mark.gpu


def _seconds(fn):
    t = time.perf_counter()
    fn()
    return time.perf_counter() - t


def _steps(x, n):
    x.step(n)
    x.sync()


# 24 pipelined runs; 24 runs whose calls of several steps are resident, asked
# for single steps; a large run that steps pipelined when asked for many
@pytest.mark.parametrize("kind", ["pipelined", "one_step", "large_run"])
def test_first_steps_do_not_wait_for_graphs(gpu, kind):
    """The launch-per-step graphs are captured with the plan (0.4 to 1.5 ms for
    these): a first call costs its uploads and cold caches more than a later
    one (0.05 to 0.35 ms)."""
    extra = []
    for rep in range(4):
        if kind == "large_run":
            p = _params(gpu, 150000, 150000, 512, False)
            x = gpu.Run(p, seed=3)
            call = lambda: x.zeitschritte(20)  # noqa: E731
        else:
            p = _params(gpu, 1600, 1500, 128 if kind == "pipelined" else 96, False)
            x = gpu.Batch([p] * 24, list(range(24)))
            call = (lambda: _steps(x, 20)) if kind == "pipelined" else (lambda: _steps(x, 1))  # noqa: E731
        x.sync()
        first = _seconds(call)
        later = min(_seconds(call) for _ in range(3))
        extra.append(first - later)
        x.close()
    bound = 0.2e-3 if kind == "one_step" else 0.7e-3
    assert min(extra) < bound, "first call %s ms longer" % ", ".join("%.2f" % (e * 1e3) for e in extra)


def test_first_sync_allocates_no_pinned_pages(gpu):
    """The run states' way to the host shares the position copies' pinned
    memory: a first synchronising call after the upload of a run whose staging
    buffer is megabytes long takes as long as a later one (0.03 ms; a pinned
    allocation of its own 1.3 to 2.9)."""
    took = []
    for rep in range(4):
        r = gpu.Run(_params(gpu, 150000, 150000, 512, False), seed=3)
        took.append(_seconds(r.sync))
        r.close()
    assert min(took) < 0.7e-3, "first sync %s ms" % ", ".join("%.2f" % (e * 1e3) for e in took)


def test_phase_times_of_a_run_that_steps_with_the_stage_kernels(gpu):
    """300 000 particles on 4096^2: steps in the stage kernels' launches; the
    pipelined step's phases can still be timed, and the steps around them have
    the bits of stage kernels throughout."""
    p = _params(gpu, 200000, 100000, 4096, False, rho=0.1)
    start = _lattice(p, 3)
    a, b = gpu.Run(p, seed=6), gpu.Run(p, seed=6)
    for r in (a, b):
        r.set_positions_all(start)
    assert a.launches_per_step() > 6
    a.zeitschritte(2)
    ms = a.fused_phase_times(3)
    assert ms is not None and sum(ms.values()) > 0.0
    a.zeitschritte(2)
    b.stage_times(7)
    x, y = a.get_positions(), b.get_positions()
    for s in (0, 1):
        assert (x[s][0] == y[s][0]).all() and (x[s][1] == y[s][1]).all()
    assert a.step_count() == b.step_count() == 7
