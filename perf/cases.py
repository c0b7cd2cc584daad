"""The solves this framework is measured on, and their 64-bit values.

Each case is a dict of plain values; ``prepare`` builds what a program holds
before the call (models, observed data, an engine or posterior), ``run`` is
one pass through the framework's public entry points, ``work`` the bytes and
operations of a pass, ``exact`` the same outputs in 64-bit arithmetic from
plain torch.

Kinds of case
  dropin     ``aco2d.fwi``: one model, host arrays in and out, as the reference's drivers call it
  engine     ``Fwi2dEngine.run`` on device tensors: misfit and gradient, the imaging condition,
             data only, or the exact discrete gradient
  posterior  ``Posterior.log_prob`` and its backward, as a variational inversion calls it
  uneven     ``gb_fwi2d_run_instances`` of the C ABI: inversions of different grids in one call
  engine3d   ``Fwi3dEngine.run``: 3-D misfit and gradient
"""
import configparser
import ctypes
import math
import os
import random
import tempfile

import numpy as np
import torch

from geopvi_gb300 import _native, aco2d, fwi3d
from geopvi_gb300.engine import Fwi2dEngine
from geopvi_gb300.params import Params, write_paramfile
from geopvi_gb300.posterior import Posterior

_GB = 1 << 30


def _case2d(name, kind, nz, nx, ns, nt, **kw):
    c = {"name": name, "kind": kind, "nz": nz, "nx": nx, "ns": ns, "nt": nt, "samples": 1, "pml0": 20, "Lc": 4,
         "nti": 1, "dx": 10.0, "dz": 10.0, "dt": 1e-3, "f0": 10.0, "nr": nx, "noise": 0.0, "mode": "fwi",
         "laplace": 0, "checkpoint": False, "budget_gb": 40}
    c.update(kw)
    return c


def _case3d(name, nx, ny, nz, ns, nt, **kw):
    c = {"name": name, "kind": "engine3d", "nx": nx, "ny": ny, "nz": nz, "ns": ns, "nt": nt, "samples": 1,
         "pml0": 10, "Lc": 4, "nti": 1, "dx": 10.0, "dy": 10.0, "dz": 10.0, "dt": 1e-3, "f0": 10.0, "rec_step": 4,
         "noise": 0.0, "mode": "fwi", "checkpoint": False}
    c.update(kw)
    return c


def listed():
    return [
        # The smallest calls: a toy inversion (tutorials, tests, a quick look) -- launches and latency.
        _case2d("toy", "engine", 32, 48, 2, 240, pml0=10, f0=15.0),
        # The reference example's own configuration (its config.ini), one model through the drop-in
        # module with host arrays, as the reference's serial drivers call it.
        _case2d("example_dropin", "dropin", 110, 250, 12, 2001, pml0=10, Lc=3, nti=2, dx=20.0, dz=20.0, dt=2e-3),
        # A small variational iteration: log_prob and backward of a few samples on the GPU.
        _case2d("vi_small", "posterior", 120, 250, 10, 2000, samples=3),
        # The batched variational iteration of the benchmark (200 x 400, 20 shots, nt 3000), with
        # the samples of a modest batch.
        _case2d("vi_batch", "engine", 200, 400, 20, 3000, samples=4, f0=8.0),
        # A long time axis on a large grid, checkpointed because its field would not be stored;
        # noisy (field) data, so the adjoint field is non-zero from its first step.
        _case2d("vi_checkpoint", "posterior", 300, 600, 8, 4000, dt=0.8e-3, checkpoint=True, noise=0.02),
        # Several inversions of different grids, shots and time axes in one call (a server's batch).
        _case2d("uneven", "uneven", 200, 400, 10, 1200, samples=2, instances=5, mix=7),
        # Observed-data generation: the largest grid, no gradient.
        _case2d("make_data", "engine", 400, 800, 16, 2000, mode="forward", f0=12.0),
        # Reverse-time migration: imaging condition, 12th order, rectangular cells, odd sizes,
        # every third step stored.
        _case2d("rtm_ragged", "engine", 157, 331, 9, 1501, mode="imaging", Lc=6, pml0=15, nti=3, dx=12.5, dz=8.0,
                dt=0.75e-3, nr=110, noise=0.02),
        # The exact discrete gradient (gradient checks, step-size calibration).
        _case2d("exact_gradient", "engine", 200, 400, 8, 1500, mode="exact", f0=8.0),
        # The pseudo-spectral Laplacian, on the grid of the small inversions.
        _case2d("pseudo_spectral", "engine", 100, 200, 4, 600, laplace=1, dt=0.8e-3),
        # 3-D misfit and gradient on the benchmark's cube.
        _case3d("cube_gradient", 160, 160, 160, 4, 200),
        # 3-D with odd sides, 12th order, rectangular cells, checkpoints, every second step imaged.
        _case3d("ragged3d_checkpoint", 75, 110, 61, 3, 240, Lc=6, pml0=8, nti=2, dx=10.0, dy=12.5, dz=8.0,
                checkpoint=True, noise=0.02),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cell_steps(c):
    """Padded cells times time steps, all solves and passes of a pass over the case."""
    if c["kind"] == "uneven":
        return sum(_cell_steps(i) for i in _instances(c))
    passes = 1 if c["mode"] == "forward" else 3 if c["checkpoint"] or c["mode"] == "exact" else 2
    pad = 2 * (c["pml0"] + (0 if c.get("laplace") else c["Lc"] + 1))
    n = (c["nz"] + pad) * (c["nx"] + pad) * ((c["ny"] + pad) if "ny" in c else 1)
    return n * c["nt"] * c["samples"] * c["ns"] * passes * (12 if c.get("laplace") else 1)


def draw(rng: random.Random):
    """One more case of the listed ranges."""
    kind = rng.choice(["dropin", "engine", "engine", "engine", "posterior", "posterior", "uneven", "engine3d"])
    Lc = rng.choice([3, 4, 4, 4, 5, 6])
    noise = rng.choice([0.0, 0.02])
    nti = rng.choice([1, 1, 1, 2, 3])
    if kind == "engine3d":
        side = lambda: _log_uniform(rng, 40, 150)  # noqa: E731
        c = _case3d("", side(), side(), side(), rng.randint(1, 5), _log_uniform(rng, 100, 300), Lc=Lc, nti=nti,
                    pml0=rng.randint(5, 12), dy=rng.choice([10.0, 12.5]), rec_step=rng.randint(2, 6), noise=noise,
                    mode=rng.choice(["fwi", "fwi", "forward"]), checkpoint=rng.random() < 0.3,
                    f0=float(rng.choice([10, 15])))
    else:
        nz = _log_uniform(rng, 30, 400)
        nx = max(40, int(nz * rng.uniform(1.2, 2.3)))
        h = rng.choice([5.0, 10.0, 12.5, 20.0])
        dz = rng.choice([h, h, 0.8 * h])
        c = _case2d("", kind, nz, nx, rng.randint(2, 20), _log_uniform(rng, 300, 3500), Lc=Lc, noise=noise, nti=nti,
                    pml0=rng.randint(8, 24), dx=h, dz=dz, dt=1e-4 * min(h, dz) * rng.choice([0.8, 1.0]),
                    f0=round(rng.uniform(5.0, 15.0) * 10.0 / h, 2), nr=rng.choice([nx, nx, nx // 2, nx // 3]),
                    samples=1 if kind == "dropin" else rng.randint(1, 6))
        if kind == "engine":
            c["mode"] = rng.choice(["fwi", "fwi", "imaging", "forward", "exact"])
            c["checkpoint"] = c["mode"] == "fwi" and rng.random() < 0.3
            if c["mode"] == "fwi" and rng.random() < 0.15 and nz <= 120:
                c.update(laplace=1, checkpoint=False, dt=0.7e-4 * min(h, dz))
        elif kind == "posterior":
            c["checkpoint"] = rng.random() < 0.4
        elif kind == "uneven":
            c.update(instances=rng.randint(2, 6), mix=rng.randint(0, 10 ** 6))
    del c["name"]
    while _cell_steps(c) > 3e10 or _stored_bytes(c) > 25 * _GB:
        if c["samples"] > 1:
            c["samples"] -= 1
        elif c["ns"] > 2:
            c["ns"] = max(2, int(c["ns"] * 0.7))
        else:
            c["nt"] = max(60, int(c["nt"] * 0.8))
    return c


def _stored_bytes(c):
    if c["kind"] == "uneven":
        return sum(_stored_bytes(i) for i in _instances(c))
    if c["mode"] == "forward" or c["checkpoint"]:
        return 0
    if c["mode"] == "exact":
        return _cell_steps(c) // 3 * 4
    return c["nz"] * c["nx"] * c.get("ny", 1) * 4 * (c["nt"] // c["nti"] + 1) * c["samples"] * c["ns"]


def _instances(c):
    """The inversions of an uneven batch: the case's own grid and smaller ones."""
    rng = random.Random(c["mix"])
    out = []
    for i in range(c["instances"]):
        f = 1.0 if i == 0 else rng.choice([0.5, 0.5, 0.75, 1.0])
        nz, nx = max(24, int(c["nz"] * f)), max(32, int(c["nx"] * f))
        d = {k: v for k, v in c.items() if k not in ("name", "instances", "mix")}
        d.update(kind="engine", nz=nz, nx=nx, nr=max(1, min(c["nr"], nx)), ns=max(1, int(c["ns"] * rng.uniform(0.4, 1.0))),
                 nt=max(50, int(c["nt"] * rng.uniform(0.4, 1.0))), samples=rng.randint(1, c["samples"]),
                 f0=round(c["f0"] * rng.uniform(0.7, 1.2), 2))
        out.append(d)
    return out


# ---- inputs -----------------------------------------------------------------

def _params(c):
    ns, nx, nr = c["ns"], c["nx"], c["nr"]
    ds = max(1, nx // ns)
    dr = max(1, nx // nr)
    return Params(nx=nx, nz=c["nz"], pml0=c["pml0"], Lc=c["Lc"], laplace_solver=c["laplace"], ns=ns, nt=c["nt"],
                  ds=ds, ns0=(nx - (ns - 1) * ds) // 2, depths=2, depthr=0, nr=nr, dr=dr,
                  nr0=(nx - (nr - 1) * dr) // 2 if nr < nx else 0, nt_interval=c["nti"], dx=c["dx"], dz=c["dz"],
                  dt=c["dt"], f0=c["f0"])


def _acquisition3d(c):
    nx, ny, ns = c["nx"], c["ny"], c["ns"]
    src = np.array([[(nx // 8 + i * (nx - nx // 4) // max(1, ns - 1)) % nx, ny // 4 + (i % 2) * (ny // 2), 2]
                    for i in range(ns)])
    rec = np.array([[x, y, 0] for y in range(0, ny, c["rec_step"]) for x in range(0, nx, c["rec_step"])])
    return src, rec


def _ricker(nt, dt, f0):
    """The reference's wavelet: float phase, double wavelet, stored as float."""
    dt, f0 = np.float32(dt), np.float32(f0)
    phase = np.arange(nt, dtype=np.float32) * dt - np.float32(1.0) / f0
    a = ((3.1415926 * np.float64(f0) * phase.astype(np.float64)) ** 2).astype(np.float32).astype(np.float64)
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _models(c, g, vmin, vmax):
    """(samples, nz*nx) or (samples, ny*nx*nz): a velocity increasing with depth, smooth anomalies
    and the per-cell scatter of a variational sample."""
    dims = (c["nz"], c["nx"]) if "ny" not in c else (c["ny"], c["nx"], c["nz"])
    zdim = 0 if "ny" not in c else 2
    grid = torch.meshgrid(*[torch.linspace(0, 1, n, device="cuda") for n in dims], indexing="ij")
    v = vmin + 0.75 * (vmax - vmin) * grid[zdim]
    for _ in range(4):
        r = torch.rand(len(dims) + 2, generator=g, device="cuda")
        d2 = sum((x - r[i]) ** 2 for i, x in enumerate(grid))
        v = v + (r[-1] - 0.5) * 0.25 * (vmax - vmin) * torch.exp(-d2 / (0.01 + 0.05 * r[-2]))
    scatter = torch.randn((c["samples"],) + dims, generator=g, device="cuda")
    return (v + 60.0 * scatter).clamp(vmin, vmax).reshape(c["samples"], -1).contiguous()


def _observed(c, offsets, g, amp):
    """(ns, nt, nr) records: a direct arrival and reflections on their travel-time curves, plus
    noise relative to the largest value (field data) where the case has some."""
    t = torch.arange(c["nt"], device="cuda", dtype=torch.float64)[None, :, None] * c["dt"] - 1.0 / c["f0"]
    off = offsets[:, None, :]
    out = torch.zeros((off.shape[0], c["nt"], off.shape[2]), dtype=torch.float32, device="cuda")
    depth = c["nz"] * c["dz"]
    r = torch.rand(8, generator=g, device="cuda").tolist()
    for i in range(4):
        v = 1600.0 + 450.0 * i + 200.0 * r[i]
        t0 = 0.0 if i == 0 else 2.0 * depth * (0.2 * i + 0.1 * r[4 + i]) / v
        arrive = torch.sqrt(t0 * t0 + (off / v) ** 2)
        a = (math.pi * c["f0"] * (t - arrive)) ** 2
        weight = amp * (1.0, -0.4, 0.3, -0.2)[i] / torch.sqrt(1.0 + (off + v * t0) / 100.0)
        out += (weight * (1 - 2 * a) * torch.exp(-a)).float()
    if c["noise"]:
        out += c["noise"] * out.abs().max() * torch.randn(out.shape, generator=g, device="cuda")
    return out.contiguous()


def _inputs2d(c, seed):
    p = _params(c)
    g = _generator(seed)
    vel = _models(c, g, 1500.0, 4700.0)
    xs = torch.arange(p.ns, device="cuda", dtype=torch.float64) * p.ds + p.ns0
    xr = torch.arange(p.nr, device="cuda", dtype=torch.float64) * p.dr + p.nr0
    obs = _observed(c, (xs[:, None] - xr[None, :]).abs() * c["dx"], g, 0.5)
    return p, vel, obs.reshape(-1)


def _inputs3d(c, seed):
    src, rec = _acquisition3d(c)
    g = _generator(seed)
    vel = _models(c, g, 1500.0, 3000.0)
    s = torch.as_tensor(src, device="cuda", dtype=torch.float64)
    r = torch.as_tensor(rec, device="cuda", dtype=torch.float64)
    h = torch.tensor([c["dx"], c["dy"]], device="cuda", dtype=torch.float64)
    off = (((s[:, None, :2] - r[None, :, :2]) * h) ** 2).sum(-1).sqrt()
    obs = _observed(c, off, g, 0.2)
    return src, rec, _ricker(c["nt"], c["dt"], c["f0"]), vel, obs


class _TempFile:
    """A parameter file that goes with the state that uses it."""

    def __init__(self):
        fd, self.path = tempfile.mkstemp(suffix=".txt", prefix="fwi_params_")
        os.close(fd)

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def _config(p):
    cfg = configparser.ConfigParser()
    cfg["FWI"] = {"nx": str(p.nx), "nz": str(p.nz), "pml": str(p.pml0), "Lc": str(p.Lc),
                  "laplace_slover": str(p.laplace_solver), "ns": str(p.ns), "nt": str(p.nt), "ds": str(p.ds),
                  "ns0": str(p.ns0), "depths": str(p.depths), "depthr": str(p.depthr), "nr": str(p.nr),
                  "dr": str(p.dr), "nr0": str(p.nr0), "nt_interval": str(p.nt_interval), "dx": str(p.dx),
                  "dz": str(p.dz), "dt": str(p.dt), "f0": str(p.f0)}
    return cfg


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "engine3d":
        src, rec, wavelet, vel, obs = _inputs3d(c, seed)
        p = fwi3d.Fwi3dParams(nx=c["nx"], ny=c["ny"], nz=c["nz"], nt=c["nt"], dt=c["dt"], dx=c["dx"], dy=c["dy"],
                              dz=c["dz"], pml0=c["pml0"], Lc=c["Lc"], nt_interval=c["nti"])
        eng = fwi3d.Fwi3dEngine(p, src, rec, wavelet, device="cuda", checkpoint=c["checkpoint"],
                                max_resident=c["samples"] * c["ns"])
        return {"case": c, "engine": eng, "vel": vel, "obs": obs}
    if c["kind"] == "uneven":
        parts = []
        for i, d in enumerate(_instances(c)):
            p, vel, obs = _inputs2d(d, seed * 64 + i)
            grad = torch.empty_like(vel)
            misfit = torch.empty(vel.shape[0], dtype=torch.float64, device="cuda")
            parts.append((p, vel, obs, grad, misfit))
        arr = (_native.CInstance * len(parts))(*[
            _native.CInstance(p.c(), vel.shape[0], vel.data_ptr(), obs.data_ptr(), None, grad.data_ptr(),
                              misfit.data_ptr()) for p, vel, obs, grad, misfit in parts])
        lib = _native.load()
        most = int(c["budget_gb"] * _GB // 2)
        need = int(lib.gb_fwi2d_instances_workspace_bytes(arr, len(parts), 0, 0))
        work = torch.empty(max(need, min(most, need + 2 * int(_stored_bytes(c) * 1.2 + (1 << 28)))),
                           dtype=torch.uint8, device="cuda")
        return {"case": c, "parts": parts, "arr": arr, "work": work, "lib": lib}
    p, vel, obs = _inputs2d(c, seed)
    if c["kind"] == "dropin":
        f = _TempFile()
        write_paramfile(f.path, p)
        return {"case": c, "file": f, "vel": vel[0].cpu().numpy().astype(np.float64), "obs": obs.cpu().numpy()}
    budget = int(c["budget_gb"] * _GB)
    if c["kind"] == "posterior":
        f = _TempFile()
        post = Posterior(obs.cpu().numpy(), _config(p), sigma=0.5, paramfile=f.path, device="cuda", hbm_budget=budget,
                         checkpoint=c["checkpoint"])
        return {"case": c, "file": f, "posterior": post, "x": vel.requires_grad_(True)}
    eng = Fwi2dEngine(p, device="cuda", hbm_budget=budget, checkpoint=c["checkpoint"])
    return {"case": c, "engine": eng, "vel": vel, "obs": obs}


# ---- one pass ---------------------------------------------------------------

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "dropin":
        syn, grad = aco2d.fwi(state["vel"], state["obs"], paramfile=state["file"].path)
        return {"syn": syn, "grad": grad}
    if kind == "posterior":
        x = state["x"]
        x.grad = None
        logp = state["posterior"].log_prob(x)
        logp.sum().backward()
        return {"logp": logp.detach(), "grad": x.grad}
    if kind == "uneven":
        st = state["lib"].gb_fwi2d_run_instances(
            state["arr"], len(state["parts"]), 0, 0, ctypes.c_void_p(state["work"].data_ptr()), state["work"].numel(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _native.check(st, "gb_fwi2d_run_instances")
        return {"grad": [q[3] for q in state["parts"]], "misfit": [q[4] for q in state["parts"]]}
    eng = state["engine"]
    if kind == "engine3d":
        r = eng.run(state["vel"], state["obs"], forward_only=c["mode"] == "forward")
        return {"misfit": r.misfit, "syn": r.syn} if c["mode"] == "forward" else {"misfit": r.misfit, "grad": r.grad}
    if c["mode"] == "forward":
        return {"syn": eng.run(state["vel"], state["obs"], forward_only=True).syn}
    r = eng.run(state["vel"], state["obs"], imaging=c["mode"] == "imaging", exact=c["mode"] == "exact")
    return {"grad": r.grad} if c["mode"] == "imaging" else {"misfit": r.misfit, "grad": r.grad}


def work(case):
    """Bytes: models, observed data and outputs once.  Flops: the stencil, update and imaging
    arithmetic of the cell updates of one forward and, with a gradient, one adjoint pass."""
    c = dict(case)
    if c["kind"] == "uneven":
        parts = [work(d) for d in _instances(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells = c["nz"] * c["nx"] * c.get("ny", 1)
    axes = 3 if "ny" in c else 2
    nr = c.get("nr") or (-(-c["nx"] // c["rec_step"])) * (-(-c["ny"] // c["rec_step"]))
    data = c["ns"] * c["nt"] * nr
    grad = c["mode"] != "forward"
    out = c["samples"] * cells if grad else c["samples"] * data
    if c["kind"] == "dropin":
        out += data
    passes = 2 if grad else 1
    pad = 2 * (c["pml0"] + (0 if c.get("laplace") else c["Lc"] + 1))
    n = (c["nz"] + pad) * (c["nx"] + pad) * ((c["ny"] + pad) if "ny" in c else 1)
    if c.get("laplace"):  # two real transforms of n points a step
        per = 2 * 2.5 * math.log2(n) + 8
    else:
        per = axes * (3 * c["Lc"] + 2) + 7 + (4 if grad else 0) / c["nti"]
    return {"bytes": 4.0 * (c["samples"] * cells + data + out), "flops": float(per * n * c["nt"] * c["samples"] * c["ns"] * passes)}


# ---- 64-bit values ----------------------------------------------------------

# Second-derivative weights of the reference (float32 tables) by half order.
_WEIGHTS = {
    3: (-49.0 / 18, 1.5, -0.15, 1.0 / 90),
    4: (-205.0 / 72, 1.6, -0.2, 8.0 / 315, -1.0 / 560),
    5: (-5269.0 / 1800, 5.0 / 3, -5.0 / 21, 5.0 / 126, -5.0 / 1008, 1.0 / 3150),
    6: (-5369.0 / 1800, 12.0 / 7, -15.0 / 56, 10.0 / 189, -1.0 / 112, 2.0 / 1925, -1.0 / 16632),
}


class _Scheme:
    """One time step in float64 for a batch of solves with velocities v (batch, z, [y,] x) on the
    padded grid: stencil (or spectral Laplacian), then the one-way absorbing blends axis by axis."""

    def __init__(self, v, dt, spacing, blend_spacing, Lc, pml0, laplace=0, axes=None):
        f32 = lambda a: float(np.float32(a))  # noqa: E731
        self.dt = f32(dt)
        self.h = [f32(d) for d in spacing]
        self.L = 0 if laplace else Lc + 1
        self.pml = pml0 + self.L
        self.w = [f32(x) for x in _WEIGHTS[Lc]]
        self.dims = v.shape[1:]
        self.nd = len(self.dims)
        self.axes = axes if axes is not None else list(range(self.nd))
        self.c2 = (v * self.dt) ** 2
        self.laplace = laplace
        self.inner = [n - 2 * self.L for n in self.dims]
        if laplace:
            k = []
            for n, h in zip(self.dims, self.h):
                dk = f32(1.0 / n / h)
                half = (n + 1) // 2
                k.append(np.array([f32(2 * 3.1415926 * dk * (i if i < half else n - i)) for i in range(n)]))
            self.kk = torch.as_tensor((k[0][:, None] ** 2 + k[1][None, :] ** 2).astype(np.float32).astype(np.float64),
                                      device=v.device)
        wt = np.array([f32(1.0 - i / pml0) for i in range(pml0)])
        self.bands = []
        for a in self.axes:
            for side in (0, 1):
                at = self.L if side == 0 else self.dims[a] - self.pml
                w = torch.as_tensor(wt if side == 0 else wt[::-1].copy(), device=v.device)
                w = w.reshape([1] + [pml0 if i == a else 1 for i in range(self.nd)])
                s = self._cut(v, a, at, pml0) * (self.dt / f32(blend_spacing[a]))
                t1, t2, t3 = (2 - s) * (1 - s) / 2, s * (2 - s), s * (s - 1) / 2
                taps1 = [2 * t1, 2 * t2, 2 * t3]
                taps0 = [t1 * t1, 2 * t1 * t2, t2 * t2 + 2 * t1 * t3, 2 * t2 * t3, t3 * t3]
                self.bands.append((a, at, 1 if side == 0 else -1, pml0, [w * x for x in taps1],
                                   [w * x for x in taps0], 1 - w))

    def _cut(self, f, axis, at, n):
        """Cells [at, at + n) along `axis`, the updated cells along the others."""
        for i in range(self.nd):
            f = f.narrow(i + 1, at, n) if i == axis else f.narrow(i + 1, self.L, self.inner[i])
        return f

    def core(self, f, axis=0, shift=0):
        return self._cut(f, axis, self.L + shift, self.inner[axis])

    def laplacian(self, p1):
        if self.laplace:
            return torch.fft.ifft2(-self.kk * torch.fft.fft2(p1)).real
        out = None
        for a, h in enumerate(self.h):
            d = self.w[0] * self.core(p1)
            for m in range(1, len(self.w)):
                d = d + self.w[m] * (self.core(p1, a, m) + self.core(p1, a, -m))
            d = d / (h * h)
            out = d if out is None else out + d
        return out

    def step(self, p1, p0):
        q = 2 * self.core(p1) - self.core(p0) + self.core(self.c2) * self.laplacian(p1)
        p2 = torch.nn.functional.pad(q, [self.L] * (2 * self.nd)) if self.L else q
        for a, at, d, n, t1, t0, omw in self.bands:
            e = omw * self._cut(p2, a, at, n)
            for m in range(3):
                e = e + t1[m] * self._cut(p1, a, at + d * m, n)
            for m in range(5):
                e = e - t0[m] * self._cut(p0, a, at + d * m, n)
            p2 = p2.clone() if p2.requires_grad else p2
            self._cut(p2, a, at, n).copy_(e)
        return p2


def _pad(v, pml):
    for i in range(1, v.dim()):
        n = v.shape[i]
        j = torch.arange(-pml, n + pml, device=v.device).clamp(0, n - 1)
        v = v.index_select(i, j)
    return v


def _exact2d(c, seed, want_syn):
    p, vel, obs = _inputs2d(c, seed)
    obs = obs.double().reshape(p.ns, p.nt, p.nr)
    out = {"misfit": [], "grad": [], "syn": []}
    for s in range(vel.shape[0]):
        v = vel[s].double().reshape(1, p.nz, p.nx)
        m, g, syn = (_exact_gradient if c["mode"] == "exact" else _reference_gradient)(c, p, v, obs)
        out["misfit"].append(m)
        out["grad"].append(g)
        out["syn"].append(syn if want_syn else None)
    return out


def _acq2d(p, pml):
    sx = torch.arange(p.ns, device="cuda") * p.ds + p.ns0 + pml
    rx = torch.arange(p.nr, device="cuda") * p.dr + p.nr0 + pml
    return torch.arange(p.ns, device="cuda"), pml + p.depths, sx, pml + p.depthr, rx


def _reference_gradient(c, p, v, obs):
    """Misfit, gradient in the reference's scaling (or image) and data of one model, all shots."""
    pml = p.pml
    vp = _pad(v, pml)
    sch = _Scheme(vp, p.dt, (p.dz, p.dx), (p.dx, p.dx), p.Lc, p.pml0, p.laplace_solver)
    b, sz, sx, rz, rx = _acq2d(p, pml)
    rik = _ricker(p.nt, p.dt, p.f0).astype(np.float64)
    v2 = vp[0] ** 2 * sch.dt * sch.dt
    at_src = v2[sz, sx]
    at_rec = v2[rz, rx]
    zero = torch.zeros((p.ns,) + tuple(vp.shape[1:]), dtype=torch.float64, device="cuda")
    p0, p1 = zero, zero
    imaging, forward = c["mode"] == "imaging", c["mode"] == "forward"
    syn = torch.empty((p.ns, p.nt, p.nr), dtype=torch.float64, device="cuda")
    core = lambda f: f[:, pml:pml + p.nz, pml:pml + p.nx]  # noqa: E731
    kept = {}
    for it in range(p.nt):
        p2 = sch.step(p1, p0)
        p2[b, sz, sx] += float(rik[it]) * at_src
        syn[:, it] = p2[:, rz, rx]
        if not forward and it % p.nt_interval == 0:
            kept[it] = core(p2).clone() if imaging else core(p2 - 2 * p1 + p0).clone()
        p0, p1 = p1, p2
    misfit = 0.5 * ((syn - obs) ** 2).sum()
    if forward:
        return misfit, None, syn
    res = obs if imaging else syn - obs
    acc = torch.zeros((p.ns, p.nz, p.nx), dtype=torch.float64, device="cuda")
    p0, p1 = zero, zero
    for it in range(p.nt - 1, -1, -1):
        p2 = sch.step(p1, p0)
        p2[:, rz, rx] += res[:, it] * at_rec
        if it in kept:
            acc += kept.pop(it) * core(p2)
        p0, p1 = p1, p2
    grad = acc.sum(0) * (p.nt_interval * sch.dt)
    if not imaging:
        grad = grad * (-2.0 / v[0] ** 3) / (sch.dt * sch.dt)
    return misfit, grad.reshape(-1), syn


def _exact_gradient(c, p, v, obs):
    """Misfit, dJ/dv and data of one model: every step's vector-Jacobian product by autograd."""
    pml = p.pml
    b, sz, sx, rz, rx = _acq2d(p, pml)
    rik = _ricker(p.nt, p.dt, p.f0).astype(np.float64)
    spacing = (p.dz, p.dx), (p.dx, p.dx), p.Lc, p.pml0
    vp = _pad(v, pml)
    hit = torch.zeros((p.ns,) + tuple(vp.shape[1:]), dtype=torch.float64, device="cuda")
    hit[b, sz, sx] = 1.0
    sch = _Scheme(vp, p.dt, *spacing)
    levels = [torch.zeros_like(hit), torch.zeros_like(hit)]
    for it in range(p.nt):
        levels.append(sch.step(levels[-1], levels[-2]) + hit * (float(rik[it]) * sch.dt * sch.dt * vp * vp))
    syn = torch.stack([q[:, rz, rx] for q in levels[2:]], 1)
    res = syn - obs
    inject = lambda r: torch.zeros_like(hit).index_put((b[:, None], torch.full_like(rx, rz)[None, :], rx[None, :]), r)  # noqa: E731
    lam1, lam2, gv = torch.zeros_like(hit), torch.zeros_like(hit), torch.zeros_like(vp)
    vl = vp.clone().requires_grad_(True)
    # The step is linear in (p1, p0) with coefficients of v: one graph per step, freed at once.
    for it in range(p.nt - 1, -1, -1):
        lam1 = lam1 + inject(res[:, it])
        a1 = levels[it + 1].requires_grad_(True)
        a0 = levels[it].requires_grad_(True)
        one = _Scheme(vl, p.dt, *spacing)
        out = one.step(a1, a0) + hit * (float(rik[it]) * one.dt * one.dt * vl * vl)
        d1, d0, dv = torch.autograd.grad(out, (a1, a0, vl), lam1)
        gv += dv
        lam1, lam2 = lam2 + d1, d0
        levels.pop()
    full = gv[0]
    zi = torch.arange(-pml, p.nz + pml, device="cuda").clamp(0, p.nz - 1)
    xi = torch.arange(-pml, p.nx + pml, device="cuda").clamp(0, p.nx - 1)
    grad = torch.zeros((p.nz, full.shape[1]), dtype=torch.float64, device="cuda").index_add_(0, zi, full)
    grad = torch.zeros((p.nz, p.nx), dtype=torch.float64, device="cuda").index_add_(1, xi, grad)
    return 0.5 * (res ** 2).sum(), grad.reshape(-1), syn


def _exact3d(c, seed):
    src, rec, wavelet, vel, obs = _inputs3d(c, seed)
    obs = obs.double()
    pml = c["pml0"] + c["Lc"] + 1
    ns, nt = c["ns"], c["nt"]
    forward = c["mode"] == "forward"
    b = torch.arange(ns, device="cuda")
    s = torch.as_tensor(src, device="cuda") + pml
    r = torch.as_tensor(rec, device="cuda") + pml
    misfits, grads, syns = [], [], []
    for m in range(vel.shape[0]):
        v = vel[m].double().reshape(1, c["ny"], c["nx"], c["nz"]).permute(0, 3, 1, 2).contiguous()  # z, y, x
        vp = _pad(v, pml)
        h = (c["dz"], c["dy"], c["dx"])
        sch = _Scheme(vp, c["dt"], h, h, c["Lc"], c["pml0"])
        at_src = vp[0][s[:, 2], s[:, 1], s[:, 0]] ** 2 * sch.dt * sch.dt
        zero = torch.zeros((ns,) + tuple(vp.shape[1:]), dtype=torch.float64, device="cuda")
        core = lambda f: f[:, pml:pml + c["nz"], pml:pml + c["ny"], pml:pml + c["nx"]]  # noqa: E731
        p0, p1 = zero, zero
        syn = torch.empty((ns, nt, r.shape[0]), dtype=torch.float64, device="cuda")
        kept = {}
        for it in range(nt):
            p2 = sch.step(p1, p0)
            p2[b, s[:, 2], s[:, 1], s[:, 0]] += float(wavelet[it]) * at_src
            syn[:, it] = p2[:, r[:, 2], r[:, 1], r[:, 0]]
            if not forward and it % c["nti"] == 0:
                kept[it] = core(p2 - 2 * p1 + p0).clone()
            p0, p1 = p1, p2
        res = syn - obs
        misfits.append(0.5 * (res ** 2).sum())
        syns.append(syn)
        if forward:
            continue
        acc = torch.zeros(kept[0].shape[1:], dtype=torch.float64, device="cuda")
        p0, p1 = zero, zero
        for it in range(nt - 1, -1, -1):
            p2 = sch.step(p1, p0)
            p2[:, r[:, 2], r[:, 1], r[:, 0]] += res[:, it]
            if it in kept:
                acc += (kept.pop(it) * core(p2)).sum(0)
            p0, p1 = p1, p2
        # stored p2 - 2 p1 + p0 is dt^2 times the second derivative
        grads.append((2.0 * c["nti"] / v[0] * acc).permute(1, 2, 0).reshape(-1))
    if forward:
        return {"misfit": torch.stack(misfits), "syn": torch.stack(syns)}
    return {"misfit": torch.stack(misfits), "grad": torch.stack(grads)}


def exact(case, seed):
    c = dict(case)
    if _cell_steps(c) > (3e10 if c["kind"] != "engine3d" else 1.2e10) or c["nt"] * c["samples"] > 7000:
        return None  # over about 20 seconds in 64 bits
    if c["kind"] == "engine3d":
        return _exact3d(c, seed)
    if c["kind"] == "uneven":
        each = [_exact2d(d, seed * 64 + i, False) for i, d in enumerate(_instances(c))]
        return {"grad": [torch.stack(e["grad"]) for e in each], "misfit": [torch.stack(e["misfit"]) for e in each]}
    e = _exact2d(c, seed, c["kind"] == "dropin" or c["mode"] == "forward")
    if c["kind"] == "dropin":
        return {"syn": e["syn"][0].reshape(-1), "grad": e["grad"][0]}
    if c["kind"] == "posterior":
        return {"logp": -torch.stack(e["misfit"]) / 0.5 ** 2, "grad": torch.stack(e["grad"]) / 0.5 ** 2}
    if c["mode"] == "forward":
        return {"syn": torch.stack(e["syn"]).reshape(len(e["syn"]), -1)}
    if c["mode"] == "imaging":
        return {"grad": torch.stack(e["grad"])}
    return {"misfit": torch.stack(e["misfit"]), "grad": torch.stack(e["grad"])}
