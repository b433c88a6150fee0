"""The resident step (many steps of a run in one launch) against the stage
kernels, bit for bit: every mesh class (powers of two, 3 * 2^k, other factors
of 3), fixed and adaptive dt, one cluster and the whole grid, one lane and
several lanes per particle, particles beyond a CTA's shared memory, and
batches of them. The sums are integers and every transform rounds as the
stage kernels' does, so the tolerance is zero."""
import numpy as np
import pytest

import configs as C

pytestmark = pytest.mark.gpu


def _params(gpu, n1, n2, mesh, adaptive, scheme=2, rho=0.2, **kw):
    L = max(12.0, ((n1 + n2) / rho) ** 0.5)
    return dict(C.CONFIGS["c1_cic"], N1=n1, N2=n2, L=L, FFT_samples=mesh, densGrid_Schema=scheme,
                lambda_kapillar=L / 9, f2_f1=-0.7, T=2.0, dt_max=2e-3 if adaptive else 1e-4,
                max_reisedistanz=0.1 if adaptive else 1e30, noise_kind=gpu.NOISE_DISK, **kw)


def _lattice(p, seed):
    """Sites of a square lattice in random order, each moved by up to what
    keeps pairs 0.9 apart."""
    rng = np.random.default_rng(seed)
    n, L = p["N1"] + p["N2"], p["L"]
    m = int(np.ceil(np.sqrt(n)))
    site = rng.permutation(m * m)[:n]
    x = np.mod(np.stack([site // m, site % m], 1) * (L / m) + rng.random((n, 2)) * max(0.0, L / m - 0.9), L)
    Cc = int(L / 2 ** (1 / 6))
    B = L / Cc
    git = np.minimum((x / B).astype(np.int32), Cc - 1)
    rel = np.clip(x - git * B, 0.0, np.float32(B) * (1 - 1e-6))
    return {0: (git[:p["N1"]], rel[:p["N1"]]), 1: (git[p["N1"]:], rel[p["N1"]:])}


def _same(a, b):
    for s in (0, 1):
        assert np.array_equal(a[s][0], b[s][0])
        assert np.array_equal(a[s][1], b[s][1])


# smallest and largest compiled meshes of every class, 144 and 648 through the
# run-time transform, 864 beyond the resident step; 3000 and 3001 particles on
# 128^2 either side of the cluster / grid rule
SIZES = [(40, 17, 8), (300, 201, 16), (300, 200, 24), (700, 333, 48), (1500, 1500, 128), (1500, 1501, 128),
         (1001, 999, 96), (900, 800, 144), (2000, 2500, 192), (5000, 4001, 256), (3000, 2999, 384),
         (9001, 6000, 512), (9001, 6000, 648), (9001, 6000, 768), (20000, 19999, 1024), (2000, 1000, 864)]


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("n1,n2,mesh", SIZES)
def test_resident_equals_stage_kernels(gpu, n1, n2, mesh, adaptive):
    p = _params(gpu, n1, n2, mesh, adaptive, scheme=(n1 + mesh) % 3)
    start = _lattice(p, 5)
    a, b = gpu.Run(p, seed=21), gpu.Run(p, seed=21)
    for r in (a, b):
        r.set_positions_all(start)
    a.zeitschritte(12)
    a.zeitschritt()
    a.zeitschritte(6)
    b.stage_times(19)
    _same(a.get_positions(), b.get_positions())
    assert a.time() == b.time() and a.step_count() == b.step_count()
    if adaptive:  # the last step's forces stay readable
        fa, fb = a.get_forces(), b.get_forces()
        for k in fa:
            assert np.array_equal(fa[k], fb[k])
    a.close()
    b.close()


def test_resident_beyond_shared_particles(gpu):
    """More particles per CTA than its shared memory holds (2048 on 148 SMs)."""
    p = _params(gpu, 200000, 150001, 256, False, rho=0.25)
    start = _lattice(p, 6)
    a, b = gpu.Run(p, seed=3), gpu.Run(p, seed=3)
    for r in (a, b):
        r.set_positions_all(start)
    a.zeitschritte(5)
    b.stage_times(5)
    _same(a.get_positions(), b.get_positions())


def test_resident_many_launches_and_other_steps(gpu):
    """More steps than one launch takes (1024 for a small run), and the forms
    of stepping after one another on one run."""
    p = _params(gpu, 250, 150, 32, False, scheme=1)
    start = _lattice(p, 7)
    a, b = gpu.Run(p, seed=8), gpu.Run(p, seed=8)
    for r in (a, b):
        r.set_positions_all(start)
    a.zeitschritte(1030)
    for n in (1000, 29, 1):
        b.zeitschritte(n)
    _same(a.get_positions(), b.get_positions())
    a.zeitschritte(3)
    a.stage_times(2)
    a.zeitschritt_debug(0.05)
    a.zeitschritte(4)
    b.stage_times(5)
    b.zeitschritt_debug(0.05)
    b.stage_times(4)
    _same(a.get_positions(), b.get_positions())


@pytest.mark.parametrize("adaptive", [False, True])
def test_resident_batch_equals_stage_kernels(gpu, adaptive):
    """A batch of uneven runs on clusters of several sizes, steps of both
    forms in turn (one step at a time takes the launch-per-step form)."""
    sizes = [(400, 300, 64), (1000, 900, 128), (600, 601, 96), (150, 0, 32), (700, 700, 192), (300, 100, 144)]
    if not adaptive:
        sizes = [(n1, n2, m) for n1, n2, m in sizes if m & (m - 1) == 0]
    runs = [_params(gpu, n1, n2, m, adaptive and k % 2 == 0, scheme=k % 3) for k, (n1, n2, m) in enumerate(sizes)]
    if adaptive:
        runs.append(dict(runs[0], idgas_only=1))
    seeds = list(range(len(runs)))
    a, b = gpu.Batch(runs, seeds), gpu.Batch(runs, seeds)
    for x in (a, b):
        for k, p in enumerate(runs):
            x.set_positions(k, _lattice(p, 40 + k))
    a.step(9)
    a.step(1)
    a.step(20)
    b.stage_times(30)
    for k in range(len(runs)):
        _same(a.get_positions(k), b.get_positions(k))
        assert a.time(k) == b.time(k)


@pytest.mark.parametrize("mesh", [2048, 4096])
def test_large_mesh_pipelined_equals_stage_kernels(gpu, mesh):
    """One run on a mesh beyond the resident step's: the pipelined step (its
    transforms read and write global memory in their outer passes, the
    spectrum by column) against the stage kernels and, after new positions,
    again; 140 000 particles take the particle kernel's form for large runs."""
    p = _params(gpu, 80000, 60001, mesh, False, scheme=2, rho=0.05)
    start, other = _lattice(p, 11), _lattice(p, 12)
    a, b = gpu.Run(p, seed=5), gpu.Run(p, seed=5)
    assert a.launches_per_step() == 6
    for r, steps in ((a, a.zeitschritte), (b, b.stage_times)):
        r.set_positions_all(start)
        steps(4)
        r.set_positions_all(other)
        steps(3)
        r.zeitschritt()
        steps(2)
    _same(a.get_positions(), b.get_positions())
    assert a.time() == b.time()
    a.forces()
    fa = a.get_forces()
    import oracle
    o = oracle.Oracle(p, 1)
    pos = a.get_positions()
    o.set_positions(pos)
    fo = o.forces()
    for s in (0, 1):  # FP32 transforms of 2^22 points and more: 1e-5 as the parity tests
        d = np.linalg.norm(fa[("kap", s)] - fo[("kap", s)]) / np.linalg.norm(fo[("kap", s)])
        assert d <= 1e-5


def test_groups_uneven_batch_equals_stage_kernels(gpu):
    """Few runs of very uneven weight: groups of CTAs of one cooperative grid,
    the smallest run on one CTA, the largest on most of them, with step
    budgets of their own through the server."""
    sizes = [(60, 41, 16), (3000, 2501, 384), (500, 400, 64), (9000, 8000, 256)]
    runs = [_params(gpu, n1, n2, m, k != 3, scheme=2) for k, (n1, n2, m) in enumerate(sizes)]
    a, b = gpu.Batch(runs, [3, 4, 5, 6]), gpu.Batch(runs, [3, 4, 5, 6])
    for x in (a, b):
        for k, p in enumerate(runs):
            x.set_positions(k, _lattice(p, 70 + k))
    a.step(13)
    a.step(7)
    b.stage_times(20)
    for k in range(len(runs)):
        _same(a.get_positions(k), b.get_positions(k))
        assert a.time(k) == b.time(k)
    runs = [dict(p, max_reisedistanz=1e30) for p in runs]  # the server steps with a fixed dt
    srv = gpu.Server(steps_per_tick=9)
    ids = [srv.submit(p, 90 + k, 5 + 11 * k) for k, p in enumerate(runs)]
    for _ in range(1000):
        srv.tick()
        if all(srv.poll(i).state >= 2 for i in ids):
            break
    for k, p in enumerate(runs):
        r = gpu.Run(p, seed=90 + k)
        r.stage_times(5 + 11 * k)
        _same(srv.result(ids[k]), r.get_positions())


def test_resident_adaptive_beyond_shared_particles(gpu):
    p = _params(gpu, 170000, 150001, 96, True, rho=0.25)
    start = _lattice(p, 6)
    a, b = gpu.Run(p, seed=3), gpu.Run(p, seed=3)
    for r in (a, b):
        r.set_positions_all(start)
    a.zeitschritte(4)
    b.stage_times(4)
    _same(a.get_positions(), b.get_positions())


# smallest and largest mesh, meshes whose column items hold one and several
# columns, one and two CTAs per SM (256 particles per CTA on 148 SMs), and
# more than 512 scan chunks (a C of 1024 and more)
@pytest.mark.parametrize("n1,n2,mesh", [(40, 17, 8), (300, 201, 32), (1500, 1501, 128), (18900, 18988, 256),
                                        (18900, 18989, 512), (20000, 19999, 1024), (180001, 130000, 256)])
def test_one_step_calls_equal_stage_kernels(gpu, n1, n2, mesh):
    p = _params(gpu, n1, n2, mesh, False, scheme=(n1 + mesh) % 3, rho=0.2 if n1 < 100000 else 0.18)
    start = _lattice(p, 15)
    a, b = gpu.Run(p, seed=22), gpu.Run(p, seed=22)
    for r in (a, b):
        r.set_positions_all(start)
    for _ in range(4):
        a.zeitschritt()
    a.zeitschritte(3)
    a.zeitschritt()
    b.stage_times(8)
    _same(a.get_positions(), b.get_positions())
    assert a.time() == b.time() and a.step_count() == b.step_count()


@pytest.mark.parametrize("n1,n2,mesh", [(65536, 65535, 512), (65536, 65536, 512), (65536, 65536, 1024),
                                        (131072, 131072, 64)])
def test_large_single_run_forms_in_turn(gpu, n1, n2, mesh):
    """Either side of the size from which calls of several steps take the
    pipelined step; single steps, short and long calls after one another."""
    p = _params(gpu, n1, n2, mesh, False, rho=0.25)
    start = _lattice(p, 16)
    a, b = gpu.Run(p, seed=23), gpu.Run(p, seed=23)
    for r in (a, b):
        r.set_positions_all(start)
    for n in (20, 1, 7, 8, 1, 3):
        a.zeitschritte(n)
    b.stage_times(40)
    _same(a.get_positions(), b.get_positions())
    assert a.launches_per_step() == 1
    assert a.time() == b.time() and a.step_count() == b.step_count()
