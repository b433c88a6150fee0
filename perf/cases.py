"""Workloads whose speed is tracked: what a program built on this library asks
of it, through the binding's public entry points.

A simulation program holds a run (`Run`), many independent runs (`Batch`) or
a request queue (`Server`), advances it by some steps and reads the positions
back for its frame files; drop-in callers also take single steps one call at
a time and evaluate the force routines on their own positions. The sizes are
those of the named configurations (plain small, reference parameter set,
medium, large, the batched ensemble) and of the tests' radix-3 meshes; `draw`
spreads them over the same ranges.

`exact` restates the step in FP64 with torch: cell-list WCA, mesh assignment,
spectral Green's multiply, the Philox noise streams, the adaptive step bound
and re-binning.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bd-simulations_b200"))
import bdsim  # noqa: E402

TWO_PI = 2.0 * math.pi
CELL = 2.0 ** (1.0 / 6.0)  # WCA cutoff and smallest cell edge
FIXED = 1e30               # travel bound that never binds: fixed dt
NOISE = {"disk": bdsim.NOISE_DISK, "gauss": bdsim.NOISE_GAUSS}


def listed():
    return [
        # the plain small run (2000 particles, CIC 128^2) between two frames
        dict(name="small_steps", kind="run", n1=1000, n2=1000, L=100.0, scheme=1, mesh=128, lam=10.0, f2=1.0,
             T=1.0, dt=1e-4, mrd=FIXED, noise="gauss", steps=400, call="steps", upload=False),
        # a drop-in caller: positions in, one zeitschritt call per step, positions out
        dict(name="small_calls", kind="run", n1=1000, n2=1000, L=100.0, scheme=2, mesh=128, lam=10.0, f2=1.0,
             T=1.0, dt=1e-4, mrd=FIXED, noise="disk", steps=50, call="calls", upload=True),
        # the reference's shipped parameter set (384^2 mesh, opposite charges), whose main loop takes
        # adaptive steps one at a time up to the next observation point (40 of them at dt_max)
        dict(name="shipped_calls", kind="run", n1=2000, n2=2000, L=300.0, scheme=2, mesh=384, lam=25.0, f2=-1.0,
             T=24.3055555, dt=0.005, mrd=0.24, noise="disk", steps=40, call="calls", upload=False),
        # a small adaptive run on a radix-3 mesh, odd particle numbers, many steps per call
        dict(name="adaptive_steps", kind="run", n1=1501, n2=703, L=140.0, scheme=1, mesh=96, lam=12.0, f2=-0.5,
             T=2.0, dt=0.002, mrd=0.1, noise="disk", steps=160, call="steps", upload=False),
        # the medium run (65 536 particles, TSC 512^2): positions in, steps, positions out
        dict(name="medium_steps", kind="run", n1=32768, n2=32768, L=512.0, scheme=2, mesh=512, lam=64.0, f2=0.5,
             T=1.0, dt=5e-5, mrd=FIXED, noise="disk", steps=200, call="steps", upload=True),
        # a fixed-dt run on a larger radix-3 mesh (the spacing a user picks need not be a power of two)
        dict(name="radix3_steps", kind="run", n1=40003, n2=29999, L=600.0, scheme=2, mesh=768, lam=60.0, f2=0.6,
             T=1.0, dt=1e-4, mrd=FIXED, noise="gauss", steps=60, call="steps", upload=False),
        # the large run (2.1 M particles, TSC 2048^2) between two frames
        dict(name="large_steps", kind="run", n1=1048576, n2=1048576, L=2896.0, scheme=2, mesh=2048, lam=256.0,
             f2=1.0, T=1.0, dt=5e-5, mrd=FIXED, noise="disk", steps=150, call="steps", upload=False),
        # force evaluation through the drop-in routines (WCA 11, 22, 12, capillary), forces to the host
        dict(name="medium_forces", kind="forces", n1=32768, n2=32768, L=512.0, scheme=2, mesh=512, lam=64.0, f2=0.5),
        # a parameter study: some small runs stepped together, frames of all of them
        dict(name="batch_small", kind="batch", runs=24, lo=512, hi=4096, mix=11, adaptive=False, radix3=False,
             noise="disk", dt=5e-5, steps=100),
        # the batched ensemble: 256 uneven runs, per-species N log-uniform in [512, 65536]
        dict(name="batch_ensemble", kind="batch", runs=256, lo=512, hi=65536, mix=2024, adaptive=False, radix3=False,
             noise="disk", dt=5e-5, steps=400),
        # a study around the reference's shipped parameters: adaptive dt, meshes with and without a factor 3
        dict(name="batch_adaptive", kind="batch", runs=16, lo=500, hi=4000, mix=5, adaptive=True, radix3=True,
             noise="disk", dt=0.002, steps=80),
        # a served burst: requests admitted, stepped together and returned (initial positions from the server)
        dict(name="served_burst", kind="serve", requests=16, lo=512, hi=8192, mix=7, noise="disk", steps=300),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2_mesh(L, lo=64, hi=512):
    return min(max(2 ** int(round(math.log2(L / 2))), lo), hi)


def draw(rng):
    u = rng.random()
    if u < 0.45:  # single fixed-dt runs
        n1 = _logint(rng, 700, 400000)
        n2 = int(n1 * rng.uniform(0.3, 1.2)) + 1
        L = round(math.sqrt((n1 + n2) / rng.uniform(0.15, 0.26)), 2)
        mesh = _pow2_mesh(L, 64, 2048)
        if rng.random() < 0.3:
            mesh = 3 * mesh // 4
        return dict(kind="run", n1=n1, n2=n2, L=L, scheme=rng.choice((1, 2, 2, 0)), mesh=mesh, lam=round(L / 9, 3),
                    f2=round(rng.uniform(-1.0, 1.0), 3), T=1.0, dt=rng.choice((5e-5, 1e-4)), mrd=FIXED,
                    noise=rng.choice(("disk", "gauss")), steps=min(300, max(20, 30000000 // (n1 + n2))),
                    call=rng.choice(("steps", "steps", "calls")), upload=rng.random() < 0.5)
    if u < 0.65:  # single adaptive runs
        n1 = _logint(rng, 500, 12000)
        n2 = int(n1 * rng.uniform(0.3, 1.2)) + 1
        L = round(math.sqrt((n1 + n2) / rng.uniform(0.04, 0.15)), 2)
        return dict(kind="run", n1=n1, n2=n2, L=L, scheme=rng.choice((1, 2)), mesh=rng.choice((64, 96, 128, 192, 256, 384)),
                    lam=round(L / 12, 3), f2=round(rng.uniform(-1.0, 1.0), 3), T=round(rng.uniform(1.0, 25.0), 2),
                    dt=rng.choice((0.002, 0.005)), mrd=0.24, noise="disk", steps=rng.randrange(30, 120),
                    call=rng.choice(("steps", "calls")), upload=False)
    if u < 0.8:  # force evaluations
        n1 = _logint(rng, 1000, 250000)
        n2 = int(n1 * rng.uniform(0.3, 1.2)) + 1
        L = round(math.sqrt((n1 + n2) / rng.uniform(0.15, 0.26)), 2)
        return dict(kind="forces", n1=n1, n2=n2, L=L, scheme=rng.choice((1, 2)), mesh=_pow2_mesh(L, 64, 1024),
                    lam=round(L / 9, 3), f2=round(rng.uniform(0.1, 1.0), 3))
    adaptive = rng.random() < 0.3
    runs = _logint(rng, 3, 16 if adaptive else 96)
    hi = _logint(rng, 1500, 4000 if adaptive else 40000)
    return dict(kind="batch", runs=runs, lo=512, hi=hi, mix=rng.randrange(1 << 20), adaptive=adaptive,
                radix3=adaptive, noise=rng.choice(("disk", "gauss")), dt=0.002 if adaptive else 5e-5,
                steps=rng.randrange(40, 160))


# ---------------------------------------------------------------------------
def _params(c, **kw):
    """Reference parameter names of one run."""
    p = dict(N1=c["n1"], N2=c["n2"], L=c["L"], densGrid_Schema=c["scheme"], FFT_samples=c["mesh"],
             lambda_kapillar=c["lam"], kapillar_vorfaktor=TWO_PI, T=c.get("T", 1.0), dt_max=c.get("dt", 5e-5),
             max_reisedistanz=c.get("mrd", FIXED), f2_f1=c["f2"], noise_kind=NOISE[c.get("noise", "disk")])
    p.update(kw)
    return p


def _mix(c):
    """The runs of a batch or of a served burst: area fraction 0.2, mesh near
    L/2, schemes in turn; the adaptive study is as sparse as the shipped set."""
    rng = np.random.default_rng(c["mix"])
    out = []
    for r in range(c.get("runs", c.get("requests"))):
        n = int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        if c.get("adaptive"):
            L = math.sqrt(2 * n / 0.06)
            mesh = (96, 128, 192, 256, 384, 64)[r % 6] if c["radix3"] else _pow2_mesh(L)
            out.append(dict(n1=n, n2=n, L=L, scheme=1 + r % 2, mesh=mesh, lam=L / 12, f2=-1.0, T=10.0, dt=c["dt"],
                            mrd=0.24, noise=c["noise"]))
        else:
            L = math.sqrt(2 * n * math.pi / (4 * 0.2))
            out.append(dict(n1=n, n2=n, L=L, scheme=r % 3 if c["kind"] == "batch" else 1 + r % 2, mesh=_pow2_mesh(L),
                            lam=L / 8, f2=1.0, T=1.0, dt=c.get("dt", 5e-5), mrd=FIXED, noise=c["noise"]))
    return out


def _start(n1, n2, L, seed):
    """Positions without overlaps, uncorrelated with the particle index: sites
    of a square lattice taken at random, each moved at random within what
    keeps pairs 0.9 apart, wrapped into the box at a random shift. In the
    reference's layout: cells int32[N][2], offsets double[N][2]."""
    rng = np.random.default_rng(seed)
    n = n1 + n2
    m = int(math.ceil(math.sqrt(n)))
    a = L / m
    site = rng.permutation(m * m)[:n]
    amp = max(0.0, a - 0.9)
    x = np.stack([site // m, site % m], 1) * a + rng.random((n, 2)) * amp + rng.random(2) * L
    x = np.mod(x, L)
    C = int(L / CELL)
    B = L / C
    git = np.minimum((x / B).astype(np.int32), C - 1)
    rel = np.clip(x - git * B, 0.0, np.nextafter(np.float32(B), np.float32(0)))
    # the library holds offsets in FP32: start from values it holds exactly
    rel = rel.astype(np.float32).astype(np.float64)
    return {0: (git[:n1].copy(), rel[:n1].copy()), 1: (git[n1:].copy(), rel[n1:].copy())}


def _buffers(n1, n2):
    return {s: (np.zeros((max(n, 1), 2), np.int32), np.zeros((max(n, 1), 2))) for s, n in ((0, n1), (1, n2))}


def _noise_seed(seed, k=0):
    return (int(seed) * 7919 + 104729 * k + 17) % (1 << 62)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "forces"):
        pos = _start(case["n1"], case["n2"], case["L"], seed)
        run = bdsim.Run(_params(case, startpos_methode=2), seed=_noise_seed(seed))
        run.set_positions_all(pos)
        run.sync()
        return {"case": case, "run": run, "pos": pos, "out": _buffers(case["n1"], case["n2"])}
    mix = _mix(case)
    if kind == "batch":
        batch = bdsim.Batch([_params(q, startpos_methode=3) for q in mix], [_noise_seed(seed, k) for k in range(len(mix))])
        for k, q in enumerate(mix):
            batch.set_positions(k, _start(q["n1"], q["n2"], q["L"], seed * 1000 + k))
        batch.sync()
        n = sum(q["n1"] + q["n2"] for q in mix)
        out = (np.zeros((n, 2), np.int32), np.zeros((n, 2)))
        views, at = [], 0
        for q in mix:  # both species of every run, one after the other
            v = []
            for m in (q["n1"], q["n2"]):
                v += [ctypes.c_void_p(out[0][at:].ctypes.data), ctypes.c_void_p(out[1][at:].ctypes.data)]
                at += m
            views.append(v)
        return {"case": case, "batch": batch, "out": out, "views": views}
    server = bdsim.Server(steps_per_tick=100)
    return {"case": case, "server": server, "seed": _noise_seed(seed),
            "requests": [_params(q, startpos_methode=1) for q in mix]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        r = state["run"]
        if case["upload"]:
            r.set_positions_all(state["pos"])
        if case["call"] == "calls":
            t = 0.0
            for _ in range(case["steps"]):
                t += r.zeitschritt()
        else:
            t = r.zeitschritte(case["steps"])
        p = r.get_positions(state["out"])
        return [p[0][0], p[0][1], p[1][0], p[1][1], t]
    if kind == "forces":
        f = state["run"].forces()
        return [f[(k, s)] for k in ("wca", "kap") for s in (0, 1)]
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        lib = bdsim.lib()
        for k, v in enumerate(state["views"]):
            st = lib.bd_batch_get_positions_all(b.h, k, *v)
            if st != 0:
                raise bdsim.BdError(st, "bd_batch_get_positions_all")
        return [state["out"][0], state["out"][1]]
    srv = state["server"]
    ids = [srv.submit(p, state["seed"] + k, case["steps"] + 10 * (k % 5)) for k, p in enumerate(state["requests"])]
    while srv.tick() or any(srv.poll(i).state < 2 for i in ids):
        pass
    git, rel = [], []
    for i in ids:
        q = srv.result(i)
        for s in (0, 1):
            git.append(q[s][0])
            rel.append(q[s][1])
        srv.release(i)
    return [np.concatenate(git), np.concatenate(rel)]


def work(case):
    """Per step: every particle's record in and out once (32 bytes); three
    real mesh transforms, assignment and interpolation stencils, the pairs of
    the 3x3 cells. Per pass also the positions to the host (and from it)."""
    def one(q, steps, io):
        n, z = q["n1"] + q["n2"], q["mesh"]
        pairs = 9 * CELL * CELL * n / (q["L"] * q["L"])
        stencil = (1, 4, 9)[q["scheme"]]
        flops = 7.5 * z * z * 2 * math.log2(z) / 2 + n * (20 * pairs + 12 * stencil + 100)
        return steps * 32.0 * n + io * 24.0 * n, steps * flops

    kind = case["kind"]
    if kind == "run":
        b, f = one(case, case["steps"], 2 if case["upload"] else 1)
    elif kind == "forces":
        b, f = one(case, 1, 1)
    else:
        got = [one(q, case["steps"], 1) for q in _mix(case)]
        b, f = sum(x[0] for x in got), sum(x[1] for x in got)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# FP64 restatement of the step with torch.
_M32 = 0xFFFFFFFF


def _philox(pid, step, att, seed):
    """Philox4x32-10 (Salmon et al., SC11), counter (pid, step, step >> 32,
    attempt), key the 64-bit seed: four int64 tensors of 32-bit words."""
    c = [pid, torch.full_like(pid, step & _M32), torch.full_like(pid, (step >> 32) & _M32), torch.full_like(pid, att)]
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        a, b = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [((b >> 32) & _M32) ^ c[1] ^ k0, b & _M32, ((a >> 32) & _M32) ^ c[3] ^ k1, a & _M32]
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c


def _noise(kind, n, step, seed, dev):
    pid = torch.arange(n, device=dev)
    if kind == "gauss":
        c = _philox(pid, step, 0, seed)
        rad = torch.sqrt(-2.0 * torch.log(((c[0] >> 8) + 1).double() * 2.0 ** -24))
        ang = TWO_PI * (c[1] >> 8).double() * 2.0 ** -24
        return torch.stack([rad * torch.cos(ang), rad * torch.sin(ang)], 1)
    out = torch.zeros(n, 2, dtype=torch.float64, device=dev)
    todo, att = pid, 0
    while len(todo):
        c = _philox(todo, step, att, seed)
        done = torch.zeros(len(todo), dtype=torch.bool, device=dev)
        for h in (0, 1):
            a = 2 * (c[2 * h] >> 9) + 1 - (1 << 23)
            b = 2 * (c[2 * h + 1] >> 9) + 1 - (1 << 23)
            ok = (a * a + b * b <= (1 << 46)) & ~done
            out[todo[ok]] = torch.stack([a[ok], b[ok]], 1).double() * (math.sqrt(5.0) * 2.0 ** -23)
            done |= ok
        todo, att = todo[~done], att + 1
    return out


class _Exact:
    """One run in FP64: cell index and in-cell offset of every particle."""

    def __init__(self, q, pos, seed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.q, self.seed, self.step, self.t = q, seed, 0, 0.0
        self.L, self.Z = q["L"], q["mesh"]
        self.C = int(self.L / CELL)
        self.B = self.L / self.C
        self.n1, self.n = q["n1"], q["n1"] + q["n2"]
        self.git = torch.from_numpy(np.concatenate([pos[0][0], pos[1][0]]).astype(np.int64)).to(self.dev)
        self.off = torch.from_numpy(np.concatenate([pos[0][1], pos[1][1]])).to(self.dev)
        self.w = torch.ones(self.n, dtype=torch.float64, device=self.dev)
        self.w[self.n1:] = q["f2"]
        Z, dx = self.Z, self.L / self.Z
        k = torch.arange(Z, dtype=torch.float64, device=self.dev)
        k = torch.where(k < Z // 2, k, k - Z)
        ph = TWO_PI * k / Z  # q dx
        s = 4 * torch.sin(0.5 * ph) ** 2 / dx / dx
        den = s[:, None] + s[None, :] + 1.0 / q["lam"] ** 2
        G = TWO_PI / den
        if q["lam"] > 0.2 * self.L:
            G[0, 0] = 0.0
        d = torch.sin(ph) / dx
        self.kx, self.ky = 1j * d[:, None] * G, 1j * d[None, :] * G
        self.dx = dx

    def wca(self):
        """Pair forces within the 3x3 cells, force 24 (2 r^-14 - r^-8) d capped at 1e5 |d|."""
        C, n = self.C, self.n
        cell = self.git[:, 0] * C + self.git[:, 1]
        order = torch.argsort(cell)
        cnt = torch.bincount(cell, minlength=C * C)
        start = torch.cumsum(cnt, 0) - cnt
        most = int(cnt.max())
        F = torch.zeros(n, 2, dtype=torch.float64, device=self.dev)
        me = torch.arange(n, device=self.dev)
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                g = torch.remainder(self.git[:, 0] + a, C) * C + torch.remainder(self.git[:, 1] + b, C)
                for m in range(most):
                    i = me[cnt[g] > m]
                    j = order[start[g[i]] + m]
                    i, j = i[i != j], j[i != j]
                    d = self.off[i] - self.off[j]
                    d[:, 0] -= a * self.B
                    d[:, 1] -= b * self.B
                    if C < 7:
                        d -= self.L * torch.round(d / self.L)
                    r2 = (d * d).sum(1)
                    ok = r2 <= CELL * CELL
                    i, d, r2 = i[ok], d[ok], r2[ok]
                    f = torch.clamp(24.0 * r2 ** -4 * (2.0 * r2 ** -3 - 1.0), max=1e5)
                    F.index_add_(0, i, f[:, None] * d)
        return F

    def mesh(self):
        Z, scheme = self.Z, self.q["scheme"]
        u = (self.git.double() * self.B + self.off) / self.dx
        k = torch.floor(u)
        d = u - k - 0.5
        if scheme == 2:
            w = [0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2]
        elif scheme == 1:
            w = [torch.clamp(-d, min=0.0), 1.0 - d.abs(), torch.clamp(d, min=0.0)]
        else:
            w = [torch.zeros_like(d), torch.ones_like(d), torch.zeros_like(d)]
        k = k.long()
        rho = torch.zeros(Z * Z, dtype=torch.float64, device=self.dev)
        taps = []
        for a in (0, 1, 2):
            for b in (0, 1, 2):
                at = torch.remainder(k[:, 0] + a - 1, Z) * Z + torch.remainder(k[:, 1] + b - 1, Z)
                wt = w[a][:, 0] * w[b][:, 1]
                rho.index_add_(0, at, wt * self.w / self.dx ** 2)
                taps.append((at, wt))
        X = torch.fft.fft2(rho.view(Z, Z))
        H = torch.stack([torch.fft.ifft2(self.kx * X).real.reshape(-1), torch.fft.ifft2(self.ky * X).real.reshape(-1)], 1)
        F = sum(wt[:, None] * H[at] for at, wt in taps) * self.w[:, None]
        if scheme == 0:  # the reference's nearest-point interpolation leaves species 2 without a y force
            F[self.n1:, 1] = 0.0
        return F

    def advance(self, steps):
        q = self.q
        for _ in range(steps):
            F = self.wca() + self.mesh()
            xi = _noise(q["noise"], self.n, self.step, self.seed, self.dev)
            dt = q["dt"]
            if q["mrd"] < 1e20:  # largest dt that keeps every component's move below the travel bound
                u = xi * math.sqrt(0.5 * q["T"]) / F
                a = q["mrd"] / F.abs()
                bound = (a / (torch.sqrt(u * u + a) + u.abs())) ** 2
                bound = torch.where(F.abs() < 1e-5, q["mrd"] ** 2 / (2.0 * q["T"] * xi * xi), bound)
                dt = min(dt, float(bound.min()))
            self.off = self.off + dt * F + math.sqrt(2.0 * q["T"] * dt) * xi
            k = torch.floor(self.off / self.B)
            self.off = self.off - k * self.B
            self.git = torch.remainder(self.git + k.long(), self.C)
            self.t += dt
            self.step += 1

    def rel(self):
        return self.off.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":  # the server draws its own initial positions
        return None
    if kind == "batch":
        mix = _mix(case)
        n = sum(q["n1"] + q["n2"] for q in mix)
        if case["steps"] * (len(mix) * 5e-3 + n * 1.5e-7) > 20.0:
            return None
        rel = []
        for k, q in enumerate(mix):
            e = _Exact(q, _start(q["n1"], q["n2"], q["L"], seed * 1000 + k), _noise_seed(seed, k))
            e.advance(case["steps"])
            rel.append(e.rel())
        return [None, np.concatenate(rel)]
    pos = _start(case["n1"], case["n2"], case["L"], seed)
    e = _Exact(case, pos, _noise_seed(seed))
    n1 = case["n1"]
    if kind == "forces":
        return [f[s].cpu().numpy() for f in (e.wca(), e.mesh()) for s in (slice(None, n1), slice(n1, None))]
    if case["steps"] * (5e-3 + (case["n1"] + case["n2"]) * 4e-8) > 20.0:
        return None
    e.advance(case["steps"])
    r = e.rel()
    return [None, r[:n1], None, r[n1:], e.t]
