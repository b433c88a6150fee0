"""Batches and served mixes with more runs than fit on the device at once in
the resident forms, of runs that have no pipelined step (adaptive dt, meshes
with a factor 3, ideal gas), against the stage kernels, bit for bit."""
import pytest

from test_gpu_resident import _lattice, _params, _same

pytestmark = pytest.mark.gpu


def _runs(gpu, n, kind):
    out = []
    for k in range(n):
        n1, n2 = 20 + k % 7, 10 + k % 3
        if kind == "adaptive":
            p = _params(gpu, n1, n2, (8, 16, 24)[k % 3], True, scheme=k % 3)
        elif kind == "radix3":
            p = _params(gpu, n1, n2, (12, 24, 18)[k % 3], False, scheme=k % 3)
        else:  # one ideal-gas run among fixed-dt runs on powers of two
            p = _params(gpu, n1, n2, (8, 16)[k % 2], False, scheme=k % 3)
            if k == n // 2:
                p["idgas_only"] = 1
        out.append(p)
    return out


# either side of a CTA of the group kernel per run (148 SMs), of the barrier
# words (256), of the cluster kernel's two CTAs per SM (296), and well beyond
@pytest.mark.parametrize("kind", ["adaptive", "radix3", "idgas"])
@pytest.mark.parametrize("n", [148, 149, 256, 257, 296, 297, 300, 420])
def test_many_runs_step(gpu, n, kind):
    runs = _runs(gpu, n, kind)
    a, b = gpu.Batch(runs, list(range(n))), gpu.Batch(runs, list(range(n)))
    for x in (a, b):
        for k, p in enumerate(runs):
            x.set_positions(k, _lattice(p, k))
    a.step(3)
    a.step(1)
    a.step(2)
    a.sync()
    b.stage_times(6)
    for k in range(n):
        _same(a.get_positions(k), b.get_positions(k))
        assert a.time(k) == b.time(k)


def test_many_served_runs(gpu):
    runs = _runs(gpu, 310, "radix3")
    srv = gpu.Server(steps_per_tick=8)
    ids = [srv.submit(p, 500 + k, 10 + k % 4) for k, p in enumerate(runs)]
    for _ in range(200):
        srv.tick()
        if all(srv.poll(i).state >= 2 for i in ids):
            break
    for k in (0, 1, 2, 150, 309):
        r = gpu.Run(runs[k], seed=500 + k)
        r.stage_times(10 + k % 4)
        _same(srv.result(ids[k]), r.get_positions())
