"""Single ideal-gas runs either side of the sizes at which calls of one step
and of several change between the resident step and the stage kernels."""
import pytest

from test_gpu_resident import _lattice, _params, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("n", [6000, 6001, 65536, 65537])
def test_ideal_gas_forms_in_turn(gpu, n, adaptive):
    p = _params(gpu, n - n // 3, n // 3, 32, adaptive, idgas_only=1)
    start = _lattice(p, 5)
    a, b = gpu.Run(p, seed=21), gpu.Run(p, seed=21)
    for r in (a, b):
        r.set_positions_all(start)
    for k in (7, 1, 18):
        if k == 1:
            a.zeitschritt()
        else:
            a.zeitschritte(k)
    a.sync()
    b.stage_times(26)
    _same(a.get_positions(), b.get_positions())
    assert a.time() == b.time() and a.step_count() == b.step_count() == 26


@pytest.mark.parametrize("n,one", [(6000, 1), (6001, 0), (200000, 0)])
def test_ideal_gas_calls_of_one_step(gpu, n, one):
    """A run of more particles than that steps with the stage kernels' launches
    (particles or forces and move, counts, scan, scatter) when asked for one."""
    r = gpu.Run(_params(gpu, n, 0, 32, False, idgas_only=1), seed=1)
    assert (r.launches_per_step() == 1) == bool(one)
