"""The work a user of the atmosphere solver has it do, as cases that can be timed and compared.

Sizes are X x Y x Z in the library's layout (Y vertical, idx = x + y*X + z*X*Y). Every case goes
through the public entry points: Environment (init, update_gpu, read_async, run_stage,
get_param_array), Ensemble and the C ABI's skt_diffuse_noalloc.

Kinds of cases:
  step      update_gpu on a sky with clouds, rain, snow and hail (plain or mixed projection)
  frame     a step and the readback of the sky fields that a viewer shows, into pinned memory
  ensemble  one step of several members of uneven sizes
  diffuse   the diffusion stage of one field (run_stage 0)
  advect    the PPM advection stage of one field (run_stage 1)
  project   density, projection and velocity correction (run_stage 3) of an injected wind
  noalloc   the diffusion of caller-owned device buffers (skt_diffuse_noalloc)
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from skewtcloudsim_gb300 import FIELDS, Ensemble, Environment, SktError, SolverConfig, _lib

SKY = ("th", "qv", "qw", "qc", "qr", "qs", "qi", "u", "v", "w", "p", "rho")
FRAME = SKY[:-1]  # the eleven fields of the reference's per-frame readback
MEMBER = ("th", "qv", "qw", "qr", "u", "v", "w", "p")
KAPPA = 287.0528 / 1003.5
RSD = 287.0528
STAGE_DIFFUSE, STAGE_ADVECT, STAGE_PROJECT = 0, 1, 3


# ---- the cases ----------------------------------------------------------------------------------

def listed():
    return [
        # an interactive frame on the reference's own compile-time grid: step, then show
        dict(name="frame-32x32x32", kind="frame", x=32, y=32, z=32, voxel=64.0, dt=0.5, mixed=False, graph=False, hills=False, tune=False),
        # the small documented workload, stepped as a captured graph
        dict(name="plain-64x32x64", kind="step", x=64, y=32, z=64, voxel=100.0, dt=0.5, mixed=False, graph=True, hills=False, tune=False),
        # a grid nobody rounded up to a multiple of four, default settings
        dict(name="plain-90x51x75-ragged", kind="step", x=90, y=51, z=75, voxel=64.0, dt=0.5, mixed=False, graph=False, hills=False, tune=False),
        # terrain: the ground is a heightfield with hills
        dict(name="plain-128x64x128-hills", kind="step", x=128, y=64, z=128, voxel=100.0, dt=0.5, mixed=False, graph=True, hills=True, tune=False),
        # the medium documented workload, default launch shapes
        dict(name="plain-256x128x256", kind="step", x=256, y=128, z=256, voxel=100.0, dt=0.5, mixed=False, graph=True, hills=False, tune=False),
        # the benchmark's workload with the reference's solver, default launch shapes
        dict(name="plain-512x256x512", kind="step", x=512, y=256, z=512, voxel=100.0, dt=0.5, mixed=False, graph=True, hills=False, tune=False),
        # the benchmark's workload with the mixed-precision solver, launch shapes from the tuner
        dict(name="mixed-512x256x512", kind="step", x=512, y=256, z=512, voxel=100.0, dt=0.5, mixed=True, graph=True, hills=False, tune=True),
        # members of the batched-ensemble configuration's sizes, each with its own sky
        dict(name="ensemble-8", kind="ensemble", members="64x32x64,96x64x96,128x64x128,64x32x64,192x96x192,96x64x96,128x64x128,64x32x64",
             voxel=100.0, dt=0.5, mixed=True),
        # single stages: theta's diffusion (the ground face differs from the other fields)
        dict(name="diffuse-theta-256x128x256", kind="diffuse", x=256, y=128, z=256, voxel=100.0, dt=0.5, field="th", sweeps=20),
        # vapour carried by a fast wind: three Courant substeps
        dict(name="advect-qv-192x96x192", kind="advect", x=192, y=96, z=192, voxel=100.0, dt=8.0, field="qv", wind=30.0),
        # the mixed projection alone
        dict(name="project-256x128x256", kind="project", x=256, y=128, z=256, voxel=100.0, dt=0.5),
        # a host framework diffusing a field in its own buffers, over hills
        dict(name="noalloc-qv-128x64x128", kind="noalloc", x=128, y=64, z=128, voxel=100.0, dt=0.5, field="qv", sweeps=20, hills=True),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "frame", "ensemble", "diffuse", "advect", "project", "noalloc"])

    def grid(lo, hi, even):
        """About lo..hi cells, wider than high; even: sizes that halve down to a small coarse grid."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        side = (2.0 * n) ** (1.0 / 3.0)
        x, y, z = (side * rng.uniform(0.7, 1.4) for _ in range(3))
        y *= 0.5
        if even:
            unit = 8 if n < 2.0e5 else 16 if n < 1.6e6 else 32
            x, y, z = (max(unit, int(v / unit + 0.5) * unit) for v in (x, y, z))
        else:
            x, y, z = (max(12, int(v)) for v in (x, y, z))
            if rng.random() < 0.5:
                x = max(12, x // 4 * 4)
        return x, y, z

    voxel, dt = rng.choice([50.0, 64.0, 100.0]), rng.choice([0.25, 0.5, 1.0])
    if kind == "ensemble":
        sizes = [rng.choice(["64x32x64", "96x64x96", "128x64x128", "192x96x192"]) for _ in range(rng.randint(3, 8))]
        return dict(kind=kind, members=",".join(sizes), voxel=100.0, dt=dt, mixed=True)
    if kind == "frame":
        x, y, z = grid(8.0e3, 3.0e5, False)
        return dict(kind=kind, x=x, y=y, z=z, voxel=voxel, dt=dt, mixed=False, graph=rng.random() < 0.5, hills=False, tune=False)
    if kind == "noalloc":
        x, y, z = grid(2.0e4, 1.4e6, False)
        while x * y * z > 2_000_000:
            z = max(12, z * 3 // 4)
        return dict(kind=kind, x=x, y=y, z=z, voxel=voxel, dt=dt, field=rng.choice(["th", "qv", "u"]), sweeps=rng.choice([7, 20]), hills=False)
    if kind == "project":
        x, y, z = grid(6.0e4, 1.6e7, True)
        return dict(kind=kind, x=x, y=y, z=z, voxel=voxel, dt=dt)
    if kind == "diffuse":
        x, y, z = grid(2.0e4, 3.0e7, False)
        return dict(kind=kind, x=x, y=y, z=z, voxel=voxel, dt=dt, field=rng.choice(["th", "qv", "u", "w"]), sweeps=rng.choice([7, 20, 20]))
    if kind == "advect":
        x, y, z = grid(2.0e4, 3.0e7, False)
        return dict(kind=kind, x=x, y=y, z=z, voxel=100.0, dt=rng.choice([0.5, 4.0, 8.0]), field=rng.choice(["th", "qv", "qw"]), wind=rng.choice([10.0, 30.0]))
    mixed = rng.random() < 0.5
    x, y, z = grid(2.0e4, 2.5e7, mixed)
    hills = not mixed and rng.random() < 0.3
    return dict(kind=kind, x=x, y=y, z=z, voxel=voxel, dt=dt, mixed=mixed, graph=rng.random() < 0.6, hills=hills, tune=not hills and rng.random() < 0.3)


# ---- inputs ---------------------------------------------------------------------------------------

def _profile(y, voxel, rng):
    """A moist sounding as level columns: theta (K), qv (kg/kg), pressure (hPa), u and w (m/s), temperature."""
    h = np.arange(y, dtype=np.float64) * voxel
    ts, lapse, top = rng.uniform(296.0, 304.0), rng.uniform(6.0e-3, 7.0e-3), 11000.0
    t = ts - lapse * np.minimum(h, top)
    tt, expo = ts - lapse * top, 9.8076 / (RSD * lapse)
    p = 1000.0 * (np.maximum(ts - lapse * np.minimum(h, top), 1.0) / ts) ** expo
    p = np.where(h < top, p, p * np.exp(-9.8076 * (h - top) / (RSD * tt)))
    es = 6.1078 * np.exp(17.27 * (t - 273.15) / (t - 273.15 + 237.3))
    rh = np.interp(h, [0.0, 2000.0, 6000.0, 1.0e5], [0.95, 0.9, 0.3, 0.3])
    qv = rh * 0.622 * es / (p - es)
    theta = t * (1000.0 / p) ** KAPPA
    u, w = rng.uniform(5.0, 10.0) * np.clip(h / 3000.0, 0.0, 1.0), rng.uniform(-2.0, 2.0) * np.clip(h / 4000.0, 0.0, 1.0)
    return theta, qv, p, u, w, t


def _hills(x, y, z, rng):
    ax, az = np.arange(x)[None, :] / x, np.arange(z)[:, None] / z
    f = 0.5 + 0.5 * np.sin(2 * math.pi * (ax + rng.random())) * np.sin(2 * math.pi * (az + rng.random()))
    return np.floor(f * max(1.0, y / 6.0)).astype(np.int32).reshape(-1)


class _Sky:
    """The fields of one sky on the GPU, shape (Z, Y, X), and the level columns."""

    def __init__(self, case, x, y, z, seed):
        rng = np.random.default_rng([int(seed), x, y, z])
        vox = case["voxel"]
        self.x, self.y, self.z, self.voxel = x, y, z, vox
        th, qv, p, u, w, t = (c.astype(np.float32) for c in _profile(y, vox, rng))
        self.cols = dict(th=th, qv=qv, p=p, u=u, w=w)
        self.heights = _hills(x, y, z, rng) if case.get("hills") else np.zeros(x * z, np.int32)
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
        dev = dict(device="cuda", dtype=torch.float32)

        def full(col):
            return torch.from_numpy(col).cuda()[None, :, None].expand(z, y, x).contiguous()

        def noise(a, size):
            return a.add_(torch.rand((z, y, x), generator=g, **dev).sub_(0.5), alpha=2.0 * size)

        xs, hs, zs = (torch.arange(n, **dev) * vox for n in (x, y, z))
        blob = torch.zeros((z, y, x), **dev)
        for _ in range(max(2, min(12, x * z // 4096))):  # warm bubbles, each with a cloud
            r = rng.uniform(0.08, 0.16) * min(x, z) * vox
            gx, gh, gz = (torch.exp(-((a - c) / s) ** 2) for a, c, s in (
                (xs, rng.uniform(0, x * vox), r), (hs, rng.uniform(0.1, 0.6) * y * vox, 0.35 * y * vox * rng.uniform(0.5, 1.0)), (zs, rng.uniform(0, z * vox), r)))
            blob += gz[:, None, None] * gh[None, :, None] * gx[None, None, :]
        self.f = f = {}
        f["th"] = noise(full(th).add_(blob, alpha=2.0), 0.05)
        f["qv"] = noise(full(qv), 2.0e-5).clamp_(min=0.0)
        f["p"] = full(p)
        for name, size in (("u", 0.3), ("v", 0.2), ("w", 0.3)):
            f[name] = noise(full(self.cols[name]) if name in self.cols else torch.zeros((z, y, x), **dev), size)
        f["v"].add_(blob, alpha=1.0)
        # condensate inside the bubbles: water and rain below the freezing level, ice and snow above
        warm = torch.from_numpy((t > 273.15).astype(np.float32)).cuda()[None, :, None]
        core = (blob - 0.35).clamp_(min=0.0)
        f["qw"] = core * 1.5e-3
        f["qr"] = (core - 0.2).clamp_(min=0.0) * 1.0e-3
        f["qc"] = core * (1.0 - warm) * 6.0e-4
        f["qs"] = (core - 0.1).clamp_(min=0.0) * (1.0 - warm) * 5.0e-4
        f["qi"] = (core - 0.3).clamp_(min=0.0) * (1.0 - warm) * 4.0e-4
        if torch.from_numpy(self.heights).any():
            sky = torch.arange(y, device="cuda")[None, :, None] > torch.from_numpy(self.heights).cuda().view(z, 1, x)
        else:
            sky = (torch.arange(y, device="cuda") > 0)[None, :, None]
        self.sky = sky
        for name in f:
            if name != "p":
                f[name].mul_(sky)

    def host(self, name):
        """A level column spread over the grid, as the host array that init takes."""
        return np.ascontiguousarray(np.broadcast_to(self.cols[name][None, :, None], (self.z, self.y, self.x))).reshape(-1)


class _Device:
    """A field of an environment as a CUDA array: the library's own buffer, as getParamArray hands it out.
    A tensor made from it keeps it, and so the environment that owns the buffer."""

    def __init__(self, env, name):
        self.env = env
        self.__cuda_array_interface__ = dict(shape=(env.nz, env.ny, env.nx), typestr="<f4", data=(env.get_param_array(*FIELDS[name]), False), version=3)


def _views(env, names):
    return {n: torch.as_tensor(_Device(env, n), device="cuda") for n in names}


def _environment(case, x, y, z, seed, cfg):
    """An environment initialised from the level columns, then given the sky's fields through its device pointers."""
    s = _Sky(case, x, y, z, seed)
    env = Environment(x, y, z, s.voxel, cfg)
    vel = np.zeros((z, y, x, 3), np.float32)
    vel[..., 0], vel[..., 2] = s.cols["u"][None, :, None], s.cols["w"][None, :, None]
    env.init(s.host("th"), vel.reshape(-1), s.host("qv"), np.full(x * z, 300.0, np.float32), np.full(x * z, 1000.0, np.float32), s.host("p"),
             s.cols["p"], s.heights, noise=False)
    for n, a in _views(env, tuple(k for k in s.f if k != "p")).items():
        a.copy_(s.f[n])
    torch.cuda.synchronize()
    return env, s


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "ensemble":
        envs = []
        for i, m in enumerate(case["members"].split(",")):
            x, y, z = (int(v) for v in m.split("x"))
            envs.append(_environment(case, x, y, z, seed * 64 + i, SolverConfig(precision=int(case["mixed"]), use_graph=1))[0])
        st.update(envs=envs, ens=Ensemble(envs), out=[_views(e, MEMBER) for e in envs])
        return st
    x, y, z = case["x"], case["y"], case["z"]
    if kind == "noalloc":
        s = _Sky(case, x, y, z, seed)
        flat = {"in": s.f[case["field"]].reshape(-1), "p": s.f["p"].reshape(-1), "gh": torch.from_numpy(s.heights).cuda(),
                "col": torch.from_numpy(s.cols[case["field"]]).cuda(), "Tg": torch.full((x * z,), 301.0, device="cuda"),
                "Pg": torch.full((x * z,), 1000.0, device="cuda"), "out": torch.empty(x * y * z, device="cuda")}
        st.update(buf=flat, lib=_lib.load())
        return st
    if kind in ("step", "frame"):
        cfg = SolverConfig(precision=int(case["mixed"]), use_graph=int(case["graph"]))
    elif kind == "project":
        cfg = SolverConfig(precision=1)
    elif kind == "diffuse":
        cfg = SolverConfig(diffuse_sweeps=case["sweeps"])
    else:
        cfg = SolverConfig()
    env, s = _environment(case, x, y, z, seed, cfg)
    st.update(env=env)
    if kind == "frame":
        st["host"] = {n: torch.empty(env.n, dtype=torch.float32, pin_memory=True) for n in FRAME}
        st["arrays"] = {n: a.numpy() for n, a in st["host"].items()}
    elif kind == "advect":
        v = _views(env, ("u", "v", "w"))
        for n, share in (("u", 1.0), ("v", 0.3), ("w", -0.7)):  # a wind of both signs, its largest value 0.98 times the named one
            v[n].copy_(_wind(s, n, case["wind"] * share))
        torch.cuda.synchronize()
        st["out"] = _views(env, (case["field"],))
    elif kind == "project":
        st["wind"] = {n: s.f[n].clone() for n in ("u", "v", "w")}
        st["out"] = _views(env, ("u", "v", "w", "p", "rho"))
    elif kind == "diffuse":
        st["out"] = _views(env, (case["field"],))
    else:
        st["out"] = _views(env, SKY)
    if case.get("tune"):
        env.autotune()
    return st


def _wind(s, name, size):
    """A smooth wind of both signs."""
    dev = dict(device="cuda", dtype=torch.float32)
    a, b, c = (torch.sin(2 * math.pi * (torch.arange(n, **dev) / n * k + o)) for n, k, o in ((s.x, 2, 0.1), (s.y, 1, 0.2), (s.z, 3, 0.3)))
    f = 0.3 + 0.68 * a[None, None, :] * b[None, :, None] * c[:, None, None]
    return (size * f * s.sky).contiguous()


# ---- one pass ---------------------------------------------------------------------------------------

_STAGE_FIELD = {STAGE_DIFFUSE: dict(th=0, qv=1, u=2, v=3, w=4, qw=5), STAGE_ADVECT: dict(th=0, u=1, v=2, w=3, qv=4, qw=5)}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "step":
        state["env"].update_gpu(c["dt"])
        return state["out"]
    if kind == "frame":
        env = state["env"]
        env.update_gpu(c["dt"])
        env.read_async(state["arrays"])
        env.read_wait()
        return state["host"]
    if kind == "ensemble":
        state["ens"].step(c["dt"])
        return state["out"]
    if kind == "diffuse":
        state["env"].run_stage(STAGE_DIFFUSE, _STAGE_FIELD[STAGE_DIFFUSE][c["field"]], c["dt"])
        return state["out"]
    if kind == "advect":
        state["env"].run_stage(STAGE_ADVECT, _STAGE_FIELD[STAGE_ADVECT][c["field"]], c["dt"])
        return state["out"]
    if kind == "project":
        for n, a in state["wind"].items():
            state["out"][n].copy_(a)
        torch.cuda.current_stream().synchronize()  # the library works on a stream of its own
        state["env"].run_stage(STAGE_PROJECT, 0, c["dt"])
        return state["out"]
    b = state["buf"]

    def f(n):
        return ctypes.cast(ctypes.c_void_p(b[n].data_ptr()), ctypes.POINTER(ctypes.c_float))

    status = state["lib"].skt_diffuse_noalloc(
        c["x"], c["y"], c["z"], c["voxel"], _STAGE_FIELD[STAGE_DIFFUSE][c["field"]], c["dt"], c["sweeps"], f("in"), f("out"),
        ctypes.cast(ctypes.c_void_p(b["gh"].data_ptr()), ctypes.POINTER(ctypes.c_int32)), f("col"), f("p"), f("Tg"), f("Pg"),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if status != 0:
        raise SktError(status, state["lib"].skt_last_error(None).decode())
    return {c["field"]: b["out"]}


# ---- what a pass cannot do without ------------------------------------------------------------------

def work(case):
    """Each input read once and each output written once; operations of the method (sweeps,
    passes, solver iterations at their usual counts)."""
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(math.prod(int(v) for v in m.split("x")) for m in case["members"].split(","))
    else:
        n = case["x"] * case["y"] * case["z"]
    sweep, ppm, plain, mixed, rest = 8.0, 5 * 75.0, 200 * 27.0, 18 * 90.0, 600.0
    if kind in ("step", "frame", "ensemble"):
        solver = mixed if case["mixed"] else plain
        extra = 4.0 * len(FRAME) if kind == "frame" else 0.0
        return dict(bytes=n * (4.0 * 2 * len(SKY) + extra), flops=n * (10 * (20 * sweep + ppm) + solver + rest))
    if kind in ("diffuse", "noalloc"):
        return dict(bytes=n * 8.0, flops=n * case["sweeps"] * sweep)
    if kind == "advect":
        return dict(bytes=n * 20.0, flops=n * ppm * max(1, math.ceil(0.98 * case["wind"] * case["dt"] / case["voxel"])))
    return dict(bytes=n * 4.0 * (6 + 5), flops=n * (mixed + 150.0))  # th, qv, p, u, v, w in; p, rho, u, v, w out


# ---- 64-bit values ------------------------------------------------------------------------------------

def _shift(a, dim, step, edge):
    """a's neighbour at +step (+1 or -1) along dim; outside: edge (a tensor that broadcasts to the slice)."""
    n = a.shape[dim]
    out = torch.empty_like(a)
    if step > 0:
        out.narrow(dim, 0, n - 1).copy_(a.narrow(dim, 1, n - 1))
        out.narrow(dim, n - 1, 1).copy_(edge)
    else:
        out.narrow(dim, 1, n - 1).copy_(a.narrow(dim, 0, n - 1))
        out.narrow(dim, 0, 1).copy_(edge)
    return out


def _exact_diffuse(q, sky, col, field, k, sweeps, face):
    """Jacobi sweeps of (1 + 6k) q = q0 + k sum of the neighbours, each from the sweep before;
    outside the grid the level's column, at the ground 0 (theta: its ground face below)."""
    col = col.view(1, -1, 1)
    ground = ~sky
    for _ in range(sweeps):
        total = torch.zeros_like(q)
        for dim in (0, 1, 2):
            edge = col if dim != 1 else col[:, -1:, :]
            for step in (1, -1):
                nb = _shift(q, dim, step, edge)
                gr = _shift(ground.expand_as(q), dim, step, torch.zeros((), dtype=torch.bool, device=q.device))
                nb[gr] = 0.0
                if field == "th" and dim == 1 and step == -1:
                    nb = torch.where(gr, face, nb)
                total += nb
        q = torch.where(sky, (q + k * total) / (1 + 6 * k), q)
    return q


def _flux(v, a, b, c, d, cdt):
    """The PPM flux through the face between b and c (upwind parabola with a limiter)."""
    up = v >= 0
    lo, mid, hi = torch.where(up, a, d), torch.where(up, b, c), torch.where(up, c, b)
    cour = (v * cdt).clamp(-1, 1)
    q0, q1 = torch.minimum(lo, torch.minimum(mid, hi)), torch.maximum(lo, torch.maximum(mid, hi))
    dl, dr, db = mid - lo, hi - mid, hi - lo
    lim = torch.minimum(0.5 * db.abs(), torch.minimum(dr.abs(), dl.abs()))
    s = torch.where(dl * dr > 0, torch.where(db >= 0, lim, -lim), 0.0)
    ls, rs = mid - 0.5 * s, mid + 0.5 * s
    one = torch.ones((), dtype=v.dtype, device=v.device)
    br = torch.where((rs > q1) & (rs - mid > 1e-16), (q1 - mid) / (rs - mid), one)
    bl = torch.where((ls < q0) & (mid - ls > 1e-16), (mid - q0) / (mid - ls), one)
    f = torch.minimum(one, torch.minimum(br, bl))
    r, left = mid + f * (rs - mid), mid + f * (ls - mid)
    flat = (r - mid) * (mid - left) <= 0
    r, left = torch.where(flat, mid, r), torch.where(flat, mid, left)
    lin = torch.where(cour > 0, -left - 2 * r + 3 * mid, -2 * left - r + 3 * mid)
    return v * (r + cour * lin + cour * cour * (left + r - 2 * mid))


def _exact_pass(q, vel, dim, cdt, outside, ground, one_side, one_ground, vel_low):
    """One directional pass over the sky rows, divided by the advected ones."""
    lo = ground if dim == 1 else outside
    hi = outside[:, -1:, :] if dim == 1 else outside
    own_lo, own_hi = q.narrow(dim, 0, 1), q.narrow(dim, q.shape[dim] - 1, 1)
    low = (own_lo if lo is None else lo.expand_as(own_lo)).expand_as(own_lo)
    high = (own_hi if hi is None else hi).expand_as(own_hi)
    w = torch.cat([low, low, q, high, high], dim)
    ones = torch.ones_like(q)
    l1, h1 = torch.full_like(low, one_ground if dim == 1 else one_side), torch.full_like(high, one_side)
    o = torch.cat([l1, l1, ones, h1, h1], dim)
    n = q.shape[dim]
    vl = torch.cat([vel_low.expand_as(low), vel], dim)  # the n + 1 faces
    cut = lambda a, i: a.narrow(dim, i, n + 1)  # noqa: E731
    f = _flux(vl, cut(w, 0), cut(w, 1), cut(w, 2), cut(w, 3), cdt)
    g = _flux(vl, cut(o, 0), cut(o, 1), cut(o, 2), cut(o, 3), cdt)
    return (q - cdt * (f.narrow(dim, 1, n) - f.narrow(dim, 0, n))) / (1 - cdt * (g.narrow(dim, 1, n) - g.narrow(dim, 0, n)))


def _exact_advect(case, s):
    field, vox = case["field"], case["voxel"]
    col = torch.from_numpy(s.cols[field] if field in s.cols else np.zeros(s.y, np.float32)).cuda().double()
    wind = [_wind(s, n, case["wind"] * share) for n, share in (("u", 1.0), ("v", 0.3), ("w", -0.7))]
    top = max(float(torch.maximum(w[0].abs().max(), w[1:].max())) for w in wind)
    sub = min(100, math.ceil(np.float32(np.float32(np.float32(top) * np.float32(case["dt"])) / np.float32(vox))))
    u, v, w = (a.double()[:, 1:, :] for a in wind)
    custom = field in ("th", "qv")
    out_col = col.view(1, -1, 1)[:, 1:, :] if custom else torch.zeros((1, s.y - 1, 1), dtype=torch.float64, device="cuda")
    ground = col[0].view(1, 1, 1) if custom else torch.zeros((1, 1, 1), dtype=torch.float64, device="cuda")
    one = 1.0 if custom else 0.0
    zero = torch.zeros((1, 1, 1), dtype=torch.float64, device="cuda")
    du, dw = (torch.from_numpy(s.cols[n]).cuda().double().view(1, -1, 1)[:, 1:, :] if custom else zero for n in ("u", "w"))
    q = s.f[field].double()
    a = q[:, 1:, :]
    full = case["dt"] / sub / vox
    for _ in range(sub):
        for dim, vel, low, cdt in ((2, u, du, full / 2), (1, v, zero, full / 2), (0, w, dw, full), (1, v, zero, full / 2), (2, u, du, full / 2)):
            a = _exact_pass(a, vel, dim, cdt, out_col, ground, one, one, low)
    q[:, 1:, :] = a
    return q


def _exact_project(case, s):
    """rho from the gas law, the velocity's divergence, A x = b by conjugate gradients, then p,
    rho and the velocity, on the sky rows."""
    sky = lambda a: a.double()[:, 1:, :]  # noqa: E731
    th, qv, p = sky(s.f["th"]), sky(s.f["qv"]), sky(s.f["p"])
    density = lambda p: p * 100 / (RSD * th * (p / 1000.0) ** KAPPA * (0.608 * qv + 1))  # noqa: E731
    u, v, w = (sky(s.f[n]).clone() for n in ("u", "v", "w"))
    du, dw = (torch.from_numpy(s.cols[n]).cuda().double().view(1, -1, 1)[:, 1:, :] for n in ("u", "w"))
    v[:, -1, :] = 0
    u[:, :, -1:] = du
    w[-1:] = dw
    rho = density(p)
    hm = lambda a, b: 2 / (1 / a + 1 / b)  # noqa: E731

    def faces(r):  # the harmonic mean density of each cell's upper faces; at the grid's end the cell's own
        return [hm(r, _shift(r, d, 1, r.narrow(d, r.shape[d] - 1, 1))) for d in (2, 1, 0)]

    hi = faces(rho)
    lo = [_shift(h, d, -1, rho.narrow(d, 0, 1)) for h, d in zip(hi, (2, 1, 0))]
    lo[1][:, 0, :] = 0  # the ground
    z0 = torch.zeros((), dtype=torch.float64, device="cuda")
    low_v = (_shift(u, 2, -1, du), _shift(v, 1, -1, z0), _shift(w, 0, -1, dw))
    b = sum(h * a - g * c for h, a, g, c in zip(hi, (u, v, w), lo, low_v))
    coef = lambda h: torch.where(h == 0, 0.0, -(1.225 / h).clamp(min=1.0))  # noqa: E731
    cu, cl = [coef(h) for h in hi], [coef(h) for h in lo]
    diag = -(sum(cu) + sum(cl))

    def matvec(x):
        y = diag * x
        for d, a, c in zip((2, 1, 0), cu, cl):
            n = x.shape[d] - 1
            y.narrow(d, 0, n).addcmul_(a.narrow(d, 0, n), x.narrow(d, 1, n))
            y.narrow(d, 1, n).addcmul_(c.narrow(d, 1, n), x.narrow(d, 0, n))
        return y

    x, r = torch.zeros_like(b), b.clone()
    zv = r / diag
    d, rz, stop = zv.clone(), (r * zv).sum(), 1e-11 * float(b.norm())
    for i in range(4000):
        q = matvec(d)
        alpha = rz / (d * q).sum()
        x.addcmul_(alpha, d)
        r.addcmul_(-alpha, q)
        if i % 50 == 49 and float(r.norm()) <= stop:
            break
        torch.div(r, diag, out=zv)
        new = (r * zv).sum()
        d.mul_(new / rz).add_(zv)
        rz = new
    p = p - x / 100
    rho = density(p)
    hi = faces(rho)
    for a, dim, h in ((u, 2, hi[0]), (v, 1, hi[1]), (w, 0, hi[2])):
        a += (_shift(x, dim, 1, z0) - x) / h
    out = {}
    for n, a in (("u", u), ("v", v), ("w", w), ("p", p), ("rho", rho)):
        g = s.f[n] if n in s.f else _init_density(s)
        out[n] = torch.cat([g.double()[:, :1, :], a], 1)
    return out


def _init_density(s):
    """The density that init leaves in the ground row: 0, no stage writes it."""
    return torch.zeros((s.z, s.y, s.x), device="cuda")


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("diffuse", "noalloc", "advect", "project"):
        return None  # a whole step: every stage's rounding travels through the ones after it
    n = case["x"] * case["y"] * case["z"]
    if n > (9.0e6 if kind == "project" else 4.0e7):
        return None
    s = _Sky(case, case["x"], case["y"], case["z"], seed)
    if kind == "advect":
        return {case["field"]: _exact_advect(case, s)}
    if kind == "project":
        return _exact_project(case, s)
    field = case["field"]
    k = 0.005 * case["dt"] / case["voxel"] ** 2
    face = None
    if field == "th":
        p = s.f["p"].double()
        if kind == "noalloc":
            tg = torch.full((1, 1, 1), 301.0, dtype=torch.float64, device="cuda")
        else:  # init sets the ground's temperature from the column's lowest level
            tg = float(s.cols["th"][0]) * (p[:, 1:2, :] / 1000.0) ** KAPPA
        face = tg * (1000.0 / p) ** KAPPA
    q = _exact_diffuse(s.f[field].double(), s.sky.expand(s.z, s.y, s.x), torch.from_numpy(s.cols[field]).cuda().double(), field, k, case["sweeps"], face)
    return {field: q.reshape(-1) if kind == "noalloc" else q}
