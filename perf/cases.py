"""The workloads this library is measured on, through its public Python API.

Each case is one thing that a user of the reference MATLAB code has a computer
do: one modeling shot, one modeling shot with wavefield snapshots, one RTM shot
by the three drop-in calls, a batch of shots (host buffers in and out, or a
device-resident plan), a large checkpointed RTM, a mix of jobs served by the
continuous-batching server.  Sizes are those of the repository's own
configurations (201 x 201, 301 x 601, 401 x 1201, 1201 x 4001 physical points;
served grids of 256 x 256 to 1024 x 2048; the small grids of its tests) with
records cut so that one pass stays under two seconds.

Models, wavelets and geometries are drawn from the seed: layers with gently
undulating interfaces and a Gaussian anomaly at 1500-4500 m/s, a Ricker source
below the CPML, receivers on every column at the next row -- the ranges of the
reference's drivers.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "mnad-modeling-rtm_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)


def listed():
    return [
        # the smallest call there is: a test-sized shot, nothing but latency
        {"name": "shot 96x112", "kind": "forward", "nz": 96, "nx": 112, "d": 10, "nt": 160},
        # the reference's plain modeling run: 201 x 201, 1 s, a receiver line
        {"name": "shot 201x201", "kind": "forward", "nz": 201, "nx": 201, "d": 20, "nt": 1000},
        # the same run with the wavefield after 0.3 and 0.6 s returned
        {"name": "wavefields 201x201", "kind": "fields", "nz": 201, "nx": 201, "d": 20, "nt": 700},
        # one shot of an odd-sized large model, no snapshots
        {"name": "shot 1023x2047", "kind": "forward", "nz": 1023, "nx": 2047, "d": 20, "nt": 800},
        # single-shot RTM by the drop-in calls: forward, background forward
        # with FP32 snapshots every 4 steps, adjoint with imaging
        {"name": "rtm shot 381x681", "kind": "rtm_shot", "nz": 381, "nx": 681, "d": 40, "nt": 1500, "T": 4,
         "codec": "f32"},
        # the same calls on the survey grid, BF16 snapshots, the reference's own snapshot interval
        {"name": "rtm shot 481x1281", "kind": "rtm_shot", "nz": 481, "nx": 1281, "d": 40, "nt": 1600, "T": 0,
         "codec": "bf16"},
        # generating synthetic data: a batch of modeling jobs of uneven record lengths, host buffers
        {"name": "modeling jobs 321x641", "kind": "jobs", "nz": 321, "nx": 641, "d": 40, "nt": 900, "shots": 8},
        # batched RTM of a survey line, device-resident plan, BF16 snapshots (the headline workload, shorter)
        {"name": "rtm plan 481x1281", "kind": "plan", "nz": 481, "nx": 1281, "d": 40, "nt": 800, "shots": 16, "T": 0,
         "codec": "bf16", "ckpt": 0},
        # batched RTM of small grids with FP16 snapshots (a scale and an encode per snapshot)
        {"name": "rtm plan 256x256 f16", "kind": "plan", "nz": 256, "nx": 256, "d": 20, "nt": 500, "shots": 6, "T": 0,
         "codec": "f16", "ckpt": 0},
        # large-scale RTM that checkpoints its source wavefield in FP16 and recomputes it
        {"name": "rtm checkpointed 1281x4081", "kind": "plan", "nz": 1281, "nx": 4081, "d": 40, "nt": 360, "shots": 2,
         "T": 0, "codec": "f32", "ckpt": 120},
        # a burst of mixed jobs to the server: small modeling and RTM jobs beside a medium and a large one
        {"name": "served mix", "kind": "served", "nz": 256, "nx": 256, "d": 20, "nt": 600, "rtm": 2, "model": 3,
         "wide": 1},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "fields", "rtm_shot", "jobs", "plan", "plan", "ckpt", "served"])
    d = rng.choice([10, 20, 30, 40])
    nz, nx = 2 * d + _log(rng, 48, 900), 2 * d + _log(rng, 60, 1800)
    # records between the shortest of the tests and the listed ones, fewer steps on large grids
    nt = max(150, min(_log(rng, 160, 1600), int(1.2e9 / (nz * nx))))
    if kind == "forward":
        return {"kind": kind, "nz": nz, "nx": nx, "d": d, "nt": nt}
    if kind == "fields":
        return {"kind": kind, "nz": min(nz, 500), "nx": min(nx, 700), "d": d, "nt": min(nt, 700)}
    codec = rng.choice(["f32", "bf16", "f16"])
    if kind == "rtm_shot":
        nz, nx = min(nz, 500), min(nx, 1300)
        return {"kind": kind, "nz": nz, "nx": nx, "d": d, "nt": max(nt, 240), "T": rng.choice([0, 2, 3, 4, 8]),
                "codec": codec}
    if kind == "jobs":
        return {"kind": kind, "nz": min(nz, 400), "nx": min(nx, 700), "d": d, "nt": min(nt, 900),
                "shots": rng.randint(2, 8)}
    if kind == "plan":
        return {"kind": kind, "nz": min(nz, 500), "nx": min(nx, 1300), "d": d, "nt": max(240, min(nt, 800)),
                "shots": rng.randint(2, 12), "T": rng.choice([0, 0, 4, 5]), "codec": codec, "ckpt": 0}
    if kind == "ckpt":
        return {"kind": "plan", "nz": 80 + _log(rng, 300, 1200), "nx": 80 + _log(rng, 600, 4000), "d": 40,
                "nt": rng.randint(241, 360), "shots": rng.randint(1, 2), "T": 0, "codec": "f32",
                "ckpt": rng.choice([60, 90, 120])}
    # served: launch groups of a few hundred tiles at most, whatever shares a tick
    nz, nx = rng.randint(96, 256), rng.randint(96, 256)
    return {"kind": kind, "nz": nz, "nx": nx, "d": min(d, 20), "nt": rng.randint(240, 700), "rtm": rng.randint(1, 2),
            "model": rng.randint(1, 3), "wide": rng.randint(0, 1)}


# ---------------------------------------------------------------------------
# Inputs

def _smooth(a, n):
    """n-point box average along both axes, edges replicated."""
    for ax in (0, 1):
        p = np.pad(a, [(n // 2 + 1, n // 2) if k == ax else (0, 0) for k in (0, 1)], mode="edge")
        c = np.cumsum(p, axis=ax)
        hi = np.take(c, np.arange(n, n + a.shape[ax]), axis=ax)
        lo = np.take(c, np.arange(0, a.shape[ax]), axis=ax)
        a = (hi - lo) / n
    return a


def _models(nz, nx, d, nt, rng):
    """(true, migration) velocity of a CPML-padded nz x nx grid, column-major;
    the first interface lies where a record of nt steps sees its reflection."""
    mz, mx = nz - 2 * d, nx - 2 * d
    z = np.arange(mz)[:, None] / mz
    x = np.arange(mx)[None, :] / mx
    nl = int(rng.integers(4, 9))
    tops = np.sort(np.concatenate(([min(0.12, 0.03 * nt / mz)], rng.uniform(0.15, 0.9, nl - 2))))
    vel = np.sort(rng.uniform(1550.0, 4000.0, nl))
    depth = z + min(0.03, 0.008 * nt / mz) * np.sin(2 * np.pi * (x / rng.uniform(0.3, 0.8) + rng.random()))
    v = vel[np.searchsorted(tops, depth)]
    cz, cx = rng.uniform(0.3, 0.7), rng.uniform(0.2, 0.8)
    v = v + rng.uniform(150.0, 400.0) * np.exp(-((z - cz) ** 2 + (x - cx) ** 2) / (2 * 0.08 ** 2))
    vs = _smooth(v, 15)
    pad = lambda a: np.asfortranarray(np.pad(np.clip(a, 1500.0, 4500.0), d, mode="edge"))  # noqa: E731
    return pad(v), pad(vs)


def _ricker(fc, dt, nt):
    tau = np.pi * (np.arange(nt) * dt - 1.1 / fc) * fc
    return (1 - 2 * tau ** 2) * np.exp(-tau ** 2)


H, DT = 10.0, 1e-3        # spacing (m) and time step (s): v dt / dx <= 0.45


def _shot(v, vs, d, nt, rng):
    """Source one row below the CPML, receivers on every physical column one row deeper."""
    nz, nx = v.shape
    return {"v": v, "vs": vs, "d": d, "nt": nt, "zs": float(d + 2), "xs": float(rng.integers(d + 2, nx - d)),
            "xr": np.arange(d + 1, nx - d + 1, dtype=np.float64), "zr": np.full(nx - 2 * d, float(d + 3)),
            "w": _ricker(rng.uniform(15.0, 28.0), DT, nt)}


def _inputs(case, seed):
    """The shots of a case with their kinds, on the host: [(kind, shot)]."""
    rng = np.random.default_rng(seed)
    nz, nx, d, nt, kind = case["nz"], case["nx"], case["d"], case["nt"], case["kind"]
    v, vs = _models(nz, nx, d, nt, rng)
    if kind in ("forward", "fields"):
        return [("model", _shot(v, None, d, nt, rng))]
    if kind == "rtm_shot":
        return [("rtm", _shot(v, vs, d, nt, rng))]
    if kind == "plan":
        return [("rtm", _shot(v, vs, d, nt, rng)) for _ in range(case["shots"])]
    if kind == "jobs":
        return [("model", _shot(v, None, d, nt - (37 * k) % 100, rng)) for k in range(case["shots"])]
    out = [("rtm", _shot(v, vs, d, nt - 50 * k, rng)) for k in range(case["rtm"])]
    out += [("model", _shot(v, None, d, nt - 30 * k, rng)) for k in range(case["model"])]
    out.append(("model", _shot(_models(nz, 2 * nx, d, nt, rng)[0], None, d, nt, rng)))
    if case["wide"]:
        out.append(("model", _shot(_models(2 * nz, 4 * nx, d, nt // 2, rng)[0], None, d, nt // 2, rng)))
        out.append(("model", _shot(_models(4 * nz, 8 * nx, d, nt // 3, rng)[0], None, d, nt // 3, rng)))
    return out


def _job(kind, s, T=0):
    import mnad
    return mnad.ShotJob(kind=kind, v=s["v"], vs=s["vs"], dx=H, dz=H, dt=DT, nt=s["nt"], d_pml=s["d"], zs=s["zs"],
                        xs=s["xs"], zr=s["zr"], xr=s["xr"], w=s["w"], T=T, keep_data=True)


def _keep_steps(case):
    return [max(1, int(0.43 * case["nt"])), max(2, int(0.86 * case["nt"]))]


def prepare(case, seed):
    import mnad
    shots = _inputs(case, seed)
    kind = case["kind"]
    st = {"case": case, "shots": shots}
    if kind == "served":
        st["server"] = mnad.Server(0, chunk_steps=64)
        st["jobs"] = [_job(k, s) for k, s in shots]
        return st
    st["ctx"] = mnad.Context(0)
    if kind == "rtm_shot":
        st["ctx"].set_options(snapshot_codec=case["codec"], T=case["T"])
    elif kind == "jobs":
        st["jobs"] = [_job(k, s) for k, s in shots]
    elif kind == "plan":
        st["ctx"].set_options(snapshot_codec=case["codec"], checkpoint_every=case["ckpt"], checkpoint_codec="f16")
        st["jobs"] = [_job(k, s, case["T"]) for k, s in shots]
        st["plan"] = st["ctx"].plan(st["jobs"])
    return st


def _outputs(jobs):
    return [{"data": j.data, "image": j.image, "illum": j.illum} if j.kind == "rtm" else {"data": j.data}
            for j in jobs]


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "served":
        srv = state["server"]
        for t in [srv.submit(j) for j in state["jobs"]]:
            srv.wait(t)
        return _outputs(state["jobs"])
    ctx = state["ctx"]
    if kind == "jobs":
        ctx.run_jobs(state["jobs"])
        return _outputs(state["jobs"])
    if kind == "plan":
        state["plan"].run()
        state["plan"].download()
        return {"shots": _outputs(state["jobs"]), "stack": list(state["plan"].stack())}
    s = state["shots"][0][1]
    geom = (H, s["xs"], s["xr"], H, s["zs"], s["zr"])
    if kind == "forward":
        return ctx.fwd(*geom, s["v"], DT, s["nt"], s["w"], s["d"])
    if kind == "fields":
        data, fields = ctx.fwd_fields(*geom, s["v"], DT, s["nt"], s["w"], s["d"], _keep_steps(case))
        return {"data": data, "fields": [list(fields[t]) for t in _keep_steps(case)]}
    data = ctx.fwd(*geom, s["v"], DT, s["nt"], s["w"], s["d"], ss=1)
    bg = ctx.fwd(*geom, s["vs"], DT, s["nt"], s["w"], s["d"], ss=1, indx=1)
    res = data - bg
    im = ctx.adj(H, H, s["nt"], DT, s["vs"], s["xr"], s["zr"], res, s["d"], ss=1)
    ctx.wavefield_release(1)
    return {"data": data, "background": bg, "image": im}


# ---------------------------------------------------------------------------
# What one pass cannot do without

def _propagations(case):
    """[(nz, nx, nt)] of one pass, recomputation included."""
    nz, nx, nt, kind = case["nz"], case["nx"], case["nt"], case["kind"]
    if kind in ("forward", "fields"):
        return [(nz, nx, nt)]
    if kind == "rtm_shot":
        return [(nz, nx, nt)] * 3
    if kind == "plan":
        return [(nz, nx, nt)] * ((4 if case["ckpt"] else 3) * case["shots"])
    if kind == "jobs":
        return [(nz, nx, nt - (37 * k) % 100) for k in range(case["shots"])]
    p = [(nz, nx, nt - 50 * k) for k in range(case["rtm"]) for _ in range(3)]
    p += [(nz, nx, nt - 30 * k) for k in range(case["model"])] + [(nz, 2 * nx, nt)]
    if case["wide"]:
        p += [(2 * nz, 4 * nx, nt // 2), (4 * nz, 8 * nx, nt // 3)]
    return p


def work(case):
    """Operations of the point updates (the 22 distinct stencil coefficients as
    alpha r + beta r^2 over the neighbour sums: 137 per point and step; the
    three CPML recurrences of three fields: 80 per strip point and direction),
    and the bytes of models in, records, images and stored snapshots out."""
    d, kind = case["d"], case["kind"]
    flops = nbytes = 0.0
    for nz, nx, nt in _propagations(case):
        flops += nt * (137.0 * nz * nx + 80.0 * 2 * d * (nz + nx))
        nbytes += 8.0 * nt * (nx - 2 * d)
    nint = (case["nz"] - 2 * d) * (case["nx"] - 2 * d)
    nbytes += 8.0 * case["nz"] * case["nx"] * (2 if kind in ("rtm_shot", "plan", "served") else 1)
    if kind == "fields":
        nbytes += 6 * 8.0 * case["nz"] * case["nx"]
    if kind in ("rtm_shot", "plan"):
        shots = case.get("shots", 1)
        nbytes += 16.0 * nint * shots
        if not case.get("ckpt"):
            # snapshots written once and read once; interval 6 stands for the reference's own
            nbytes += 2.0 * shots * nint * (case["nt"] // (case["T"] or 6)) * (4 if case["codec"] == "f32" else 2)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same results in 64 bits: the scheme of the reference's sources in plain torch

def _weights(dx, dz, dev):
    """alpha, beta (3 x 3 x 5 x 5, [row of U, V, W][field][z][x]): the operator
    is alpha r + beta r^2 with r = v^2 dt^2 (SRC/MNAD/A??_gen.m)."""
    A, B = np.zeros((3, 3, 5, 5)), np.zeros((3, 3, 5, 5))

    def put(r, f, dj, di, a, b):
        A[r, f, 2 + dj, 2 + di] += a
        B[r, f, 2 + dj, 2 + di] += b

    d4 = [(-1, -1), (1, -1), (-1, 1), (1, 1)]
    for s in (-1, 1):
        put(0, 0, s, 0, 24 / 11 / dz**2, -(15 / (11 * dz**4) + 1 / (dx**2 * dz**2)))
        put(0, 0, 0, s, 24 / 11 / dx**2, -(15 / (11 * dx**4) + 1 / (dx**2 * dz**2)))
        put(0, 1, 0, s, s * 20 / 33 / dx, -s * (47 / (66 * dx**3) + 1 / (6 * dx * dz**2)))
        put(0, 1, 0, 2 * s, -s / 132 / dx, s / 66 / dx**3)
        put(0, 2, s, 0, s * 20 / 33 / dz, -s * (47 / (66 * dz**3) + 1 / (6 * dz * dx**2)))
        put(0, 2, 2 * s, 0, -s / 132 / dz, s / 66 / dz**3)
        put(1, 0, 0, s, -s * (15 / (2 * dx**3) - 1 / (dx * dz**2)),
            s * (15 / (2 * dx**5) - 1 / (dx * dz**4) + 5 / (2 * dx**3 * dz**2)))
        put(2, 0, s, 0, -s * (15 / (2 * dz**3) - 1 / (dz * dx**2)),
            s * (15 / (2 * dz**5) - 1 / (dz * dx**4) + 5 / (2 * dz**3 * dx**2)))
        put(1, 1, s, 0, 1 / dz**2, -2 / (dx**2 * dz**2))
        put(1, 1, 0, s, -1.5 / dx**2, 5 / (2 * dx**4) + 1 / (2 * dx**2 * dz**2))
        put(2, 2, s, 0, -1.5 / dz**2, 5 / (2 * dz**4) + 1 / (2 * dx**2 * dz**2))
        put(2, 2, 0, s, 1 / dx**2, -2 / (dx**2 * dz**2))
    for j, i in d4:
        put(0, 0, j, i, 0, 1 / (2 * dx**2 * dz**2))
        put(0, 1, j, i, 0, i / (12 * dx * dz**2))
        put(0, 2, j, i, 0, j / (12 * dz * dx**2))
        put(1, 0, j, i, -i / (2 * dx * dz**2), -i * (5 / (4 * dx**3 * dz**2) - 1 / (2 * dx * dz**4)))
        put(2, 0, j, i, -j / (2 * dz * dx**2), -j * (5 / (4 * dz**3 * dx**2) - 1 / (2 * dz * dx**4)))
        put(1, 1, j, i, 0, -1 / (4 * dx**2 * dz**2))
        put(2, 2, j, i, 0, -1 / (4 * dx**2 * dz**2))
        put(1, 2, j, i, -i * j / (4 * dz * dx), i * j / (4 * dz**3 * dx))
        put(2, 1, j, i, -i * j / (4 * dz * dx), i * j / (4 * dx**3 * dz))
    put(0, 0, 0, 0, -48 / 11 * (1 / dx**2 + 1 / dz**2), 30 / 11 * (1 / dx**4 + 1 / dz**4 + 11 / (15 * dx**2 * dz**2)))
    put(1, 1, 0, 0, -(12 / dx**2 + 2 / dz**2), 10 / dx**4 + 4 / (dx**2 * dz**2))
    put(2, 2, 0, 0, -(12 / dz**2 + 2 / dx**2), 10 / dz**4 + 4 / (dx**2 * dz**2))
    return torch.tensor(np.concatenate([A, B]), device=dev)


class _Propagation:
    """U, V, W of one shot in 64 bits (fwd_PDE_exact_MNAD.m, Born_adj_MNAD.m)."""

    def __init__(self, v, d):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.v = torch.tensor(np.ascontiguousarray(v), device=self.dev)
        self.nz, self.nx = v.shape
        self.d = d
        self.r = (self.v * DT) ** 2
        self.k = _weights(H, H, self.dev)
        z = lambda: torch.zeros(3, self.nz + 4, self.nx + 4, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.f, self.p = z(), z()
        self.sides = []
        D = d * H
        for axis, n in ((2, self.nx), (1, self.nz)):
            for low in (True, False):
                if d == 0:
                    continue
                a = 0 if low else n - d
                X = D - H * torch.arange(d, device=self.dev, dtype=torch.float64) if low else \
                    H * torch.arange(1, d + 1, device=self.dev, dtype=torch.float64)
                X = X[None, :] if axis == 2 else X[:, None]
                vel = self.v.narrow(axis - 1, a, d)
                s0 = 3 * math.log(1e4) / (2 * D**3) * vel
                sig, dsig = s0 * X**2, 2 * s0 * X
                den = 1 + sig * DT / 2
                m = [torch.zeros(3, *vel.shape, dtype=torch.float64, device=self.dev) for _ in range(3)]
                self.sides.append((axis, a, low, (1 - sig * DT / 2) / den, dsig * DT / den, sig * DT / den, m))

    def _cpml(self):
        cp = torch.zeros(3, self.nz, self.nx, dtype=torch.float64, device=self.dev)
        inner = self.f[:, 2:-2, 2:-2]
        for axis, a, low, c1, c2, c3, m in self.sides:
            d = self.d
            f0 = inner.narrow(axis, a, d)
            wide = self.f[:, 2:-2, :] if axis == 2 else self.f[:, :, 2:-2]
            fa, fd = wide.narrow(axis, a + 3, d), wide.narrow(axis, a + 1, d)
            gr = fd - fa if low else fa - fd
            lap = fd - 2 * f0 + fa
            g = c2 / (2 * H) * gr
            m[2].mul_(c1).add_(g)
            m[1].mul_(c1).add_(2 * g + c3 * (lap / H**2 - m[2]))
            m[0].mul_(c1).add_(g + c3 * (2 * lap / H**2 - m[1]))
            cp.narrow(axis, a, d).add_(m[0])
        return cp

    def step(self, inject):
        """One step; `inject` adds to U between the CPML and the stencil (forward)."""
        cp = self._cpml()
        if inject is not None:
            self.f[0, inject[0] + 2, inject[1] + 2] += self.r[inject[0], inject[1]] * inject[2]
        with torch.backends.cudnn.flags(enabled=False):
            ab = torch.nn.functional.conv2d(self.f[None], self.k)[0]
        c = 2 * self.f[:, 2:-2, 2:-2]
        new = ab[:3] * self.r + ab[3:] * self.r**2 + c - self.p[:, 2:-2, 2:-2] - self.r * cp
        self.p[:, 2:-2, 2:-2] = new
        self.f, self.p = self.p, self.f
        return new

    def interior(self, a):
        d = self.d
        return a[d:self.nz - d, d:self.nx - d]


def _plan_of(vs, nt, T):
    nf = math.floor(nt / (2.0 * 3.0 * vs.max() / vs.min()))
    T = T or math.floor(nt / nf / 2.0)
    return T, max(2 * nf + 1, nt // T)


def _forward(s, v, T=0, keep=()):
    """Gather (nt x nr); with T the d2u snapshots and T * illumination; the fields after the listed steps."""
    P = _Propagation(v, s["d"])
    zr, xr = (torch.tensor(a.astype(np.int64) - 1, device=P.dev) for a in (s["zr"], s["xr"]))
    zs, xs = int(s["zs"]) - 1, int(s["xs"]) - 1
    data, snaps, illum, kept = [], [], 0.0, []
    for tt in range(1, s["nt"] + 1):
        old = P.p[0, 2:-2, 2:-2].clone() if T and tt % T == 0 else None
        new = P.step((zs, xs, float(s["w"][tt - 1])))
        data.append(P.p[0, zr + 2, xr + 2])                 # U of this step: after the injection, before the update
        if T and tt % T == 0:
            d2u = new[0] - (2 * P.p[0, 2:-2, 2:-2] if tt >= 2 else 0) + (old if tt >= 3 else 0)
            d2u = P.interior(d2u / DT**2)
            snaps.append(d2u.clone())
            illum = illum + d2u**2
        if tt in keep:
            kept.append([a.cpu().numpy() for a in new])
    return torch.stack(data), snaps, T * illum if T else None, kept


def _adjoint(s, vs, res, snaps, T, ncols):
    P = _Propagation(vs, s["d"])
    zr, xr = (torch.tensor(a.astype(np.int64) - 1, device=P.dev) for a in (s["zr"], s["xr"]))
    im = torch.zeros(P.nz - 2 * P.d, P.nx - 2 * P.d, dtype=torch.float64, device=P.dev)
    count = 0
    for tt in range(s["nt"], 0, -1):
        new = P.step(None)
        P.p[0, zr + 2, xr + 2] += P.r[zr, xr] * res[tt - 1]
        if tt % T == 0:
            col = ncols - count
            if col <= len(snaps):
                im += snaps[col - 1] * P.interior(new[0])
            count += 1
    return T * im


def _exact_rtm(s, T):
    T, ncols = _plan_of(s["vs"], s["nt"], T)
    data, _, _, _ = _forward(s, s["v"])
    bg, snaps, illum, _ = _forward(s, s["vs"], T)
    im = _adjoint(s, s["vs"], data - bg, snaps, T, ncols)
    host = lambda a: a.cpu().numpy()  # noqa: E731
    return {"data": host(data), "background": host(bg), "res": host(data - bg), "image": host(im), "illum": host(illum)}


def exact(case, seed):
    shots, kind = _inputs(case, seed), case["kind"]
    if kind == "forward":
        return _forward(shots[0][1], shots[0][1]["v"])[0].cpu().numpy()
    if kind == "fields":
        data, _, _, kept = _forward(shots[0][1], shots[0][1]["v"], keep=_keep_steps(case))
        return {"data": data.cpu().numpy(), "fields": kept}
    if kind == "rtm_shot":
        e = _exact_rtm(shots[0][1], case["T"])
        return {k: e[k] for k in ("data", "background", "image")}
    # batches: the first job of each kind
    out, seen = [], set()
    for k, s in shots:
        new = k not in seen
        seen.add(k)
        if k == "model":
            out.append({"data": _forward(s, s["v"])[0].cpu().numpy() if new else None})
        elif new:
            e = _exact_rtm(s, case.get("T", 0))
            out.append({"data": e["res"], "image": e["image"], "illum": e["illum"]})
        else:
            out.append({"data": None, "image": None, "illum": None})
    return {"shots": out, "stack": [None, None, None]} if kind == "plan" else out
