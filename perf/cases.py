"""Performance cases of the framework: what its users have it do, through its public entry points.

A case is one of
  step2 / step3   one time step of a 2D / 3D scene from a given particle state, state in and state out
                  (device tensors, or host arrays as the CSV driver exchanges them);
  batch           a few steps of many independent scenes, then every scene read back;
  csr             the allocation-free PPE solve on a caller's device CSR system;
  train           one epoch of training of the learned-solve network.
Scenes are the repository's own layouts (dam break, hydrostatic tank, 3D dam break) with its stock
method set, in the middle of a flow: disordered particles, a vortical velocity field, a pressure near the
hydrostatic one as the step before left it.  The PPE is solved to the default 1e-10 of |b|; where the
tolerance is relative to the initial residual (the reference's criterion, with its CG) or the condition
number is a caller's, to 1e-12, which leaves about the same error in the pressure.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openmps_gb300 import _abi as abi
from openmps_gb300 import learned, scenes
from openmps_gb300.computer import Batch, Computer, load_library, mlp_train

SOLVERS = {"cg64": abi.SOLVER_CG64, "mixed": abi.SOLVER_MIXED, "learned": abi.SOLVER_LEARNED,
           "mixed_mg": abi.SOLVER_MIXED_MG}
F2 = ("x", "z", "u", "w", "p", "n")
F3 = ("x", "y", "z", "u", "v", "w", "p", "n")


# ---------------------------------------------------------------------------------------- the cases
def _step2(name, l0, water, tank, solver, **kw):
    d = dict(kind="step2", l0=l0, water_w=water[0], water_h=water[1], tank_w=tank[0], tank_h=tank[1], re=4.0,
             solver=solver, host=False, cfl=False, gc=False, explicit=False)
    d.update(kw)
    if name:
        d["name"] = name
    return d


def listed():
    dam, dam_tank = (0.2, 0.4), (0.8, 0.6)
    return [
        # the reference's own size with its default solver, particles exchanged with host arrays every
        # step as the driver does: latency and launches count
        _step2("dam_2k_cg64_host", 1e-2, dam, dam_tank, "cg64", host=True),
        # the same scene kept on the device with the fast solver
        _step2("dam_2k_mg", 1e-2, dam, dam_tank, "mixed_mg"),
        # an ordinary design-study size, odd extents, another radius, CFL time step
        _step2("dam_17k_mg_cfl", 2.3e-3, (0.211, 0.397), (0.803, 0.601), "mixed_mg", re=3.1, cfl=True),
        # the hydrostatic tank with the reference's algorithm (plain FP64 CG) and with the fast solver
        _step2("hydrostatic_84k_cg64", 2.5e-3, (1.0, 0.5), (1.0, 0.6), "cg64"),
        _step2("hydrostatic_84k_mg", 2.5e-3, (1.0, 0.5), (1.0, 0.6), "mixed_mg"),
        # the learned warm start on a middle-sized dam break
        _step2("dam_88k_learned", 1e-3, dam, dam_tank, "learned"),
        # the headline workload
        _step2("dam_340k_mg", 5e-4, dam, dam_tank, "mixed_mg"),
        # weakly compressible run with the corrective matrix: no PPE, neighbour walks only
        _step2("dam_340k_explicit_gc", 5e-4, dam, dam_tank, "cg64", gc=True, explicit=True),
        # the 3D dam break
        dict(name="dam3d_104k_mixed", kind="step3", l0=5e-3, water_w=0.2, water_d=0.1, water_h=0.4, tank_w=0.8,
             tank_h=0.6, re=2.4, solver="mixed"),
        # the batched workload: independent dam breaks of seeded column sizes
        dict(name="batch_256", kind="batch", l0=5e-3, scenes=256, steps=10),
        # a caller with its own CSR system and no allocator
        dict(name="csr_100k", kind="csr", nx=397, nz=253, radius=3.1),
        # training of the network: 200k samples in minibatches of 4096
        dict(name="train_200k", kind="train", n=200_000, batch=4096, epochs=1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["cg64", "mixed_mg", "mixed_mg", "learned", "explicit", "step3", "batch", "csr", "train"])
    if kind in ("cg64", "mixed_mg", "learned", "explicit"):
        fluid = _log(rng, 700, 60_000 if kind == "cg64" else 300_000)
        w, h = rng.uniform(0.1, 0.3), rng.uniform(0.2, 0.5)
        l0 = math.sqrt(w * h / fluid)
        return _step2(None, l0, (w, h), (max(0.8, 2 * w), 0.6), "cg64" if kind == "explicit" else kind,
                      re=rng.choice([3.1, 3.5, 4.0]), host=rng.random() < 0.25, cfl=rng.random() < 0.25,
                      gc=rng.random() < (0.5 if kind == "explicit" else 0.15), explicit=kind == "explicit")
    if kind == "step3":
        return dict(kind="step3", l0=_log(rng, 5.2e-3, 1.5e-2), water_w=rng.uniform(0.12, 0.25), water_d=0.1,
                    water_h=rng.uniform(0.2, 0.4), tank_w=0.8, tank_h=0.6, re=2.4,
                    solver=rng.choice(["mixed", "cg64"]))
    if kind == "batch":
        return dict(kind="batch", l0=rng.uniform(5e-3, 9e-3), scenes=int(_log(rng, 12, 250)), steps=rng.randint(1, 8))
    if kind == "csr":
        n = _log(rng, 500, 120_000)
        aspect = rng.uniform(0.4, 2.5)
        return dict(kind="csr", nx=max(8, int(math.sqrt(n * aspect))), nz=max(8, int(math.sqrt(n / aspect))),
                    radius=rng.choice([1.1, 2.1, 3.1, 4.1]))
    return dict(kind="train", n=int(_log(rng, 2_000, 190_000)), batch=rng.choice([512, 1000, 2048, 4096]), epochs=1)


# ---------------------------------------------------------------------------------- scenes and states
def _flow(s, width, height, depth, rng, axes):
    """The scene in the middle of a flow: disorder of a tenth of l0, vortices, a pressure near hydrostatic."""
    fluid = s.type == abi.TYPE_FLUID
    m = int(fluid.sum())
    for a in axes:
        getattr(s, a)[fluid] += (2 * rng.random(m) - 1) * 0.1 * s.l0
    x, z = s.x[fluid], s.z[fluid]
    speed, kx, kz = 0.3, math.pi / width, math.pi / height
    px, pz = 0.5 * rng.random(), 0.5 * rng.random()
    s.u[fluid] = speed * np.sin(kx * x + px) * np.cos(kz * z + pz) + 0.01 * speed * rng.standard_normal(m)
    s.w[fluid] = -speed * kx / kz * np.cos(kx * x + px) * np.sin(kz * z + pz) + 0.01 * speed * rng.standard_normal(m)
    if "y" in axes:
        s.v[fluid] = 0.05 * speed * np.sin(2 * math.pi * s.y[fluid] / depth) + 0.01 * speed * rng.standard_normal(m)
    wet = (s.type != abi.TYPE_DUMMY) & (s.x < width + 3 * s.l0) & (s.z < height)
    wave = 1 + 0.1 * np.sin(2 * kx * s.x[wet] + 6 * px) * np.cos(kz * s.z[wet])
    s.p[wet] = 1000.0 * 9.8 * np.maximum(height - s.z[wet], 0.0) * wave
    return s


def _scene2(case, seed):
    s = scenes.dam_break(case["l0"], case["water_w"], case["water_h"], case["tank_w"], case["tank_h"])
    return _flow(s, case["water_w"], case["water_h"], 0.0, np.random.default_rng(seed), "xz")


def _scene3(case, seed):
    d = case["water_d"]
    s = scenes.dam_break3d(case["l0"], (case["water_w"], d, case["water_h"]), (case["tank_w"], d, case["tank_h"]))
    return _flow(s, case["water_w"], case["water_h"], d, np.random.default_rng(seed), "xyz")


def _batch_scenes(case, seed):
    out = []
    for k in range(case["scenes"]):
        s = scenes.batch_scene(k, l0=case["l0"])  # the workload's column sizes
        out.append(_flow(s, s.meta["water_w"], s.meta["water_h"], 0.0, np.random.default_rng([seed, k]), "xz"))
    return out


def _flags(case):
    f = abi.PRESET_REFERENCE
    if case.get("gc"):
        f |= abi.FLAG_GC
    if case.get("explicit"):
        f |= abi.FLAG_PRESSURE_EXPLICIT
    return f


SOUND = 28.0  # m/s, about ten times the largest speed


def _params(case, s, dt):
    plain = case.get("solver") == "cg64"
    tol = dict(eps=1e-12 if plain else 1e-10, criterion=abi.CRIT_INITIAL_RESIDUAL if plain else abi.CRIT_RHS)
    return s.params(**dict(scenes.STOCK_PHYSICS, re_by_l0=case.get("re", 4.0), flags=_flags(case), max_dt=dt,
                           solver=SOLVERS[case.get("solver", "mixed_mg")], sound_speed=SOUND, **tol))


def _dt(case):
    dt = case["l0"] / 20.0  # the Courant number of the workloads at l0 = 5e-4 m
    return min(dt, 0.1 * case["l0"] / SOUND) if case.get("explicit") else dt


def _csr(case, seed):
    """CSR of a PPE-like operator on an nx x nz lattice: a_ij = c_ij / r^3 within `radius` spacings, c_ij
    symmetric in [0.9, 1.1], rows summing to zero but at the free surface (top row), negative definite."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx, nz = case["nx"], case["nz"]
    n = nx * nz
    R = int(math.floor(case["radius"]))
    h = torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
    ix = torch.arange(n, device="cuda") // nz
    iz = torch.arange(n, device="cuda") % nz
    rows, cols, vals = [], [], []
    diag = torch.where(iz == nz - 1, -1.0, 0.0).to(torch.float64)
    for dx in range(-R, R + 1):
        for dz in range(-R, R + 1):
            r2 = dx * dx + dz * dz
            if r2 == 0 or r2 >= case["radius"] ** 2:
                continue
            ok = (ix + dx >= 0) & (ix + dx < nx) & (iz + dz >= 0) & (iz + dz < nz)
            i = torch.nonzero(ok).flatten()
            j = i + dx * nz + dz
            v = (0.9 + 0.1 * (h[i] + h[j])) / r2 ** 1.5
            rows.append(i)
            cols.append(j)
            vals.append(v)
            diag[i] -= v
    rows.append(torch.arange(n, device="cuda"))
    cols.append(torch.arange(n, device="cuda"))
    vals.append(diag)
    row, col, val = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    order = torch.argsort(row * n + col)
    row, col, val = row[order], col[order], val[order]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    b = torch.randn(n, device="cuda", dtype=torch.float64, generator=g)
    return ptr, col.to(torch.int32), val, b


def _samples(case, seed):
    """Training samples around the shipped network's feature statistics, and the weights to start from."""
    rng = np.random.default_rng(seed)
    blob = np.array(learned.load(), dtype=np.float32)
    f = blob[0:16] + blob[16:32] * rng.standard_normal((case["n"], 16), dtype=np.float32)
    t = (f - blob[0:16]) / blob[16:32]
    y = 0.4 * t[:, 8] + 0.2 * np.tanh(t[:, 0] + t[:, 4]) + 0.05 * rng.standard_normal(case["n"], dtype=np.float32)
    return blob, np.concatenate([f, y[:, None], t[:, 8:9]], axis=1).astype(np.float32)


# ------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step2", "step3"):
        three = kind == "step3"
        s = _scene3(case, seed) if three else _scene2(case, seed)
        dt = _dt(case)
        c = Computer(_params(case, s, dt))
        if case["solver"] == "learned":
            c.learned_set_weights(learned.load())
        c.add_scene(s)
        names = F3 if three else F2
        host = three or bool(case.get("host"))  # 3D particles are exchanged through host arrays only
        a = {k: np.ascontiguousarray(getattr(s, k)) for k in ("type",) + names}
        if host:
            out = {k: np.empty_like(v) for k, v in a.items()}
        else:
            a = {k: torch.from_numpy(v).cuda() for k, v in a.items()}
            out = {k: torch.empty_like(v) for k, v in a.items()}
        return dict(kind=kind, c=c, dt=None if case.get("cfl") else dt, host=host, a=a, out=out)
    if kind == "batch":
        sc = _batch_scenes(case, seed)
        dt = _dt(case)
        return dict(kind=kind, b=Batch(_params(case, sc[0], dt), sc), dt=dt, steps=case["steps"])
    if kind == "csr":
        ptr, col, val, b = _csr(case, seed)
        return dict(kind=kind, ptr=ptr, col=col, val=val, b=b, x=torch.empty_like(b), lib=load_library())
    blob, smp = _samples(case, seed)
    return dict(kind=kind, blob=blob, samples=smp, batch=case["batch"], epochs=case["epochs"])


def run(state):
    kind = state["kind"]
    if kind in ("step2", "step3"):
        c, a, out = state["c"], state["a"], state["out"]
        if kind == "step3":
            c.set_particles3(a["type"], *[a[k] for k in F3])
            c.forward_time(state["dt"])
            return c.particles3()
        if state["host"]:
            c.set_particles(a["type"], *[a[k] for k in F2])
            c.forward_time(state["dt"])
            c.get_particles_into(out["type"], *[out[k] for k in F2])
            return out
        c._check(c.lib.mps_set_particles_device(c.h, *[a[k].data_ptr() for k in ("type",) + F2]))
        c.forward_time(state["dt"])
        c._check(c.lib.mps_get_particles_device(c.h, *[out[k].data_ptr() for k in ("type",) + F2]))
        return out
    if kind == "batch":
        b = state["b"]
        b.forward(state["dt"], state["steps"])
        all_ = [b.scene(k) for k in range(len(b.counts))]
        return {k: np.concatenate([s[k] for s in all_]) for k in ("type",) + F2}
    if kind == "csr":
        s = state
        s["x"].zero_()
        n = s["b"].numel()
        rc = s["lib"].mps_cg_solve_csr_device_noalloc(n, s["ptr"].data_ptr(), s["col"].data_ptr(), s["val"].data_ptr(),
                                                      s["b"].data_ptr(), s["x"].data_ptr(), 1e-12, abi.CRIT_RHS, 0,
                                                      torch.cuda.current_stream().cuda_stream, None, None)
        if rc:
            raise RuntimeError("status %d" % rc)
        return s["x"]
    blob, loss = mlp_train(state["blob"], state["samples"], state["epochs"], batch=state["batch"])
    return {"blob": blob, "loss": loss}


# ------------------------------------------------------------------------------------------- the work
def _count2(case):
    n = lambda v: int(round(v / case["l0"]))
    tc, tr = n(case["tank_w"]), n(case["tank_h"])
    return n(case["water_w"]) * n(case["water_h"]), (tc + 10) * (tr + 5) - tc * tr


def work(case):
    """State in and out once (a CSR solve: the system; training: the samples) and the arithmetic of the
    neighbour sums and of the solve's matrix products."""
    kind = case["kind"]
    if kind in ("step2", "batch"):
        if kind == "batch":
            per = case["l0"] ** -2 * 0.2 * 0.35
            tc, tr = 0.8 / case["l0"], 0.6 / case["l0"]
            fluid, wall, steps = case["scenes"] * per, case["scenes"] * ((tc + 10) * (tr + 5) - tc * tr), case["steps"]
        else:
            (fluid, wall), steps = _count2(case), 1
        nb = math.pi * case.get("re", 4.0) ** 2
        its = 0 if case.get("explicit") else 3 * math.sqrt(fluid + wall) if case.get("solver") == "cg64" else 45
        return dict(bytes=104.0 * (fluid + wall), flops=steps * fluid * nb * (80 + 2 * its))
    if kind == "step3":
        n = lambda v: int(round(v / case["l0"]))
        fluid = n(case["water_w"]) * n(case["water_d"]) * n(case["water_h"])
        ext = (n(case["tank_w"]) + 6) * (n(case["water_d"]) + 6) * (n(case["tank_h"]) + 3)
        wall = ext - n(case["tank_w"]) * n(case["water_d"]) * n(case["tank_h"])
        return dict(bytes=136.0 * (fluid + wall), flops=fluid * 4 / 3 * math.pi * case["re"] ** 3 * (100 + 2 * 250))
    if kind == "csr":
        n = case["nx"] * case["nz"]
        nb = math.pi * case["radius"] ** 2
        return dict(bytes=n * (12.0 * nb + 32), flops=n * nb * 2 * 3 * math.sqrt(n))
    return dict(bytes=case["epochs"] * case["n"] * 72.0, flops=case["epochs"] * case["n"] * 6.0 * 9600)


# -------------------------------------------------------------------------- the same in plain FP64 torch
def _lattice_n0(re, l0, dim):
    """The reference's lattice number density: offsets from -ceil(re) up to but not including it."""
    k = math.ceil(re / l0 - 1e-9)
    ax = np.arange(-k, k) * l0
    d = np.meshgrid(*[ax] * dim, indexing="ij")
    r = np.sqrt(sum(c * c for c in d)).ravel()
    r = r[(r > 0) & (r < re)]
    return float((re / r - 1).sum())


def _pairs(pos, lo, nl, live, scene):
    """All ordered pairs (i, j) of live particles of one scene closer than nl."""
    dim = len(pos)
    cell = [torch.floor((c - m) / nl).to(torch.int64) + 1 for c, m in zip(pos, lo)]
    size = [int(c.max()) + 3 for c in cell]
    key = scene.clone()
    for c, m in zip(cell, size):
        key = key * m + c
    key = torch.where(live, key, torch.full_like(key, -1))
    order = torch.argsort(key)
    sorted_key = key[order]
    ids = torch.nonzero(live).flatten()
    found_i, found_j = [], []
    for off in np.ndindex(*[3] * dim):
        shift = 0
        for o, m in zip(off, size):
            shift = shift * m + (o - 1)
        want = key[ids] + shift
        a = torch.searchsorted(sorted_key, want)
        cnt = torch.searchsorted(sorted_key, want, right=True) - a
        i = torch.repeat_interleave(ids, cnt)
        first = torch.repeat_interleave(a - (torch.cumsum(cnt, 0) - cnt), cnt)
        j = order[first + torch.arange(i.numel(), device=i.device)]
        d2 = sum((c[j] - c[i]) ** 2 for c in pos)
        ok = (i != j) & (d2 < nl * nl)
        found_i.append(i[ok])
        found_j.append(j[ok])
    return torch.cat(found_i), torch.cat(found_j)


def _solve(row, col, val, diag, b, x0):
    """CG on the negative definite system to the FP64 limit."""
    n = b.numel()
    idx = torch.arange(n, device=b.device)
    r_, c_, v_ = torch.cat([row, idx]), torch.cat([col, idx]), torch.cat([-val, -diag])
    order = torch.argsort(r_ * n + c_)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=b.device)
    ptr[1:] = torch.cumsum(torch.bincount(r_, minlength=n), 0)
    A = torch.sparse_csr_tensor(ptr, c_[order], v_[order], size=(n, n))
    mul = lambda v: (A @ v[:, None])[:, 0]
    x, goal = x0.clone(), 1e-28 * float(b @ b)
    for _ in range(4):  # restarted from the true residual
        r = -b - mul(x)
        p, rr = r.clone(), r @ r
        best = float(rr)
        for it in range(20 * int(math.sqrt(n)) + 500):
            q = mul(p)
            a = rr / (p @ q)
            x += a * p
            r -= a * q
            new = r @ r
            p = r + (new / rr) * p
            rr = new
            if it % 50 == 49 and float(rr) < goal:
                break
        if best < 100 * goal:
            break
    return x


class _Flow:
    """One step of the stock method set (HS, HL, ECS, DS, SPP; with `gc` and `explicit` on request)."""

    def __init__(self, case, dim, l0, dt, lo):
        self.dim, self.l0, self.dt, self.lo = dim, l0, dt, lo
        self.re = case.get("re", 4.0) * l0
        self.n0 = _lattice_n0(self.re, l0, dim)
        self.gc, self.explicit, self.cfl = bool(case.get("gc")), bool(case.get("explicit")), bool(case.get("cfl"))
        self.rho, self.nu, self.g = 1000.0, 1e-6, 9.8

    def acc(self, i, v):
        return torch.zeros(self.N, dtype=torch.float64, device="cuda").index_add_(0, i, v)

    def geometry(self, pos):
        i, j = self.pi, self.pj
        d = [c[j] - c[i] for c in pos]
        r2 = d[0] * d[0]
        for c in d[1:]:
            r2 = r2 + c * c
        ok = r2 < self.re * self.re
        i, j, d, r2 = i[ok], j[ok], [c[ok] for c in d], r2[ok]
        r = torch.sqrt(r2)
        return i, j, d, r2, r, self.re / r - 1

    def densities(self, i, w):
        n = self.acc(i, w)
        n = torch.where(self.dummy, torch.full_like(n, self.n0), n)
        return n

    def speed(self, i, j, d, r, vel, nws):
        s = self.acc(i, sum(a * (v[j] - v[i]) for a, v in zip(d, vel)) / r ** 3)
        return torch.where(nws < self.n0, torch.zeros_like(s), -self.re * s)

    def spp(self, i, d, w, nws):
        """Offset of the space potential particle of each particle that has one."""
        gx = [self.acc(i, w * c) / self.n0 for c in d]
        rg = torch.sqrt(sum(c * c for c in gx))
        has = (nws < self.n0) & (rg > 2.220446049250313e-16) & ~self.dummy
        r = self.re / ((self.n0 - nws) + 1.0)
        safe = torch.where(has, rg, torch.ones_like(rg))
        return has, [torch.where(has, -(r / safe) * c, torch.ones_like(c)) for c in gx], torch.where(has, r, torch.ones_like(r))

    def step(self, type_, pos, vel, p, n, scene):
        self.N = type_.numel()
        self.dummy, fluid = type_ == abi.TYPE_DUMMY, type_ == abi.TYPE_FLUID
        dim, dt = self.dim, self.dt
        if self.cfl:
            top = float(torch.sqrt(sum(v * v for v in vel)).max())
            dt = min(dt, 0.1 * self.l0 / top) if top > 0 else dt
        wall = [c.clone() for c in pos]
        self.pi, self.pj = _pairs(pos, self.lo, 1.2 * self.re, torch.ones_like(fluid), scene)
        i, j, d, r2, r, w = self.geometry(pos)
        nws = self.densities(i, w)
        nd = torch.where(self.dummy, n, torch.clamp(nws, min=self.n0))
        sp = self.speed(i, j, d, r, vel, nws)
        err = (nd - self.n0) / self.n0
        ecs = err.abs() * sp + sp.abs() * err
        act = ~self.dummy[j]
        c = self.nu * (5 - dim) * self.re / self.n0 / r[act] ** 3
        grav = [0.0] * (dim - 1) + [-self.g]
        a = [self.acc(i[act], c * (v[j[act]] - v[i[act]])) + g for v, g in zip(vel, grav)]
        vel = [torch.where(fluid, v + q * dt, torch.zeros_like(v)) for v, q in zip(vel, a)]
        pos = [torch.where(fluid, x + v * dt, y) for x, v, y in zip(pos, vel, wall)]
        i, j, d, r2, r, w = self.geometry(pos)
        nws = self.densities(i, w)
        nd = torch.where(self.dummy, n, torch.clamp(nws, min=self.n0))
        act = ~self.dummy[j]
        has, off, rs = self.spp(i, d, w, nws)
        if self.explicit:
            rho = self.rho / self.n0 * nd
            p = torch.where(rho <= self.rho, torch.zeros_like(rho), SOUND ** 2 * (rho - self.rho))
        else:
            b = -self.rho / (self.n0 * dt) * (self.speed(i, j, d, r, vel, nws) + ecs)
            coef = (5 - dim) * self.re / self.n0
            pair = act & ~self.dummy[i]
            val = coef / r[pair] ** 3
            diag = -self.acc(i[pair], val) - torch.where(has, coef / rs ** 3, torch.zeros_like(rs))
            rows = torch.nonzero(~self.dummy).flatten()
            place = torch.full((self.N,), -1, dtype=torch.int64, device="cuda")
            place[rows] = torch.arange(rows.numel(), device="cuda")
            q = _solve(place[i[pair]], place[j[pair]], val, diag[rows], b[rows], p[rows])
            p = p.clone()
            p[rows] = torch.clamp(q, min=0.0)
        C = None
        if self.gc:
            m = torch.zeros(self.N, dim, dim, dtype=torch.float64, device="cuda")
            sw = torch.where(has, (self.re / rs - 1) / rs ** 2, torch.zeros_like(rs))
            for k in range(dim):
                for l in range(dim):
                    m[:, k, l] = self.acc(i, w / r2 * d[k] * d[l]) + sw * off[k] * off[l]
            m[~fluid] = torch.eye(dim, dtype=torch.float64, device="cuda")
            C = torch.linalg.inv(m)
            factor = -dt * nd / (self.rho * self.n0)
        else:
            factor = -dt / self.rho * dim / self.n0
        k = (p[j[act]] + p[i[act]]) / r2[act] * w[act]
        ks = torch.where(has, p / rs ** 2 * (self.re / rs - 1), torch.zeros_like(p))
        s = torch.stack([self.acc(i[act], k * c[act]) + ks * o for c, o in zip(d, off)], 1)
        if C is not None:
            s = torch.einsum("nkl,nl->nk", C, s)
        old = pos
        pos, vel = self.move(pos, vel, [factor * s[:, k] for k in range(dim)], fluid, dt)
        i, j, d, r2, r, w = self.geometry(pos)
        lim = (0.9 * self.l0) ** 2
        hit = (r2 < lim) & ~self.dummy[j]
        i, j, d = i[hit], j[hit], [c[hit] for c in d]
        d0 = [c[j] - c[i] for c in old]
        nrm = torch.sqrt(sum(c * c for c in d0))
        e = [c / nrm for c in d0]
        par = sum(x * y for x, y in zip(d, e))
        perp2 = sum((x - par * y) ** 2 for x, y in zip(d, e))
        mag = torch.sqrt(lim - perp2) - par
        pos, vel = self.move(pos, vel, [-1.0 / (2 * dt * self.n0) * self.acc(i, mag * c) for c in e], fluid, dt)
        return pos, vel, p, nd

    @staticmethod
    def move(pos, vel, dv, fluid, dt):
        dv = [torch.where(fluid, v, torch.zeros_like(v)) for v in dv]
        return [x + v * dt for x, v in zip(pos, dv)], [u + v for u, v in zip(vel, dv)]


def _exact_flow(case, parts, dim, lo, steps):
    cat = lambda k: torch.from_numpy(np.concatenate([getattr(s, k) for s in parts])).cuda()
    axes, vels = ("xyz", "uvw") if dim == 3 else ("xz", "uw")
    type_ = cat("type")
    pos, vel, p, n = [cat(k) for k in axes], [cat(k) for k in vels], cat("p"), cat("n")
    scene = torch.repeat_interleave(torch.arange(len(parts)), torch.tensor([s.count for s in parts])).cuda()
    flow = _Flow(case, dim, case["l0"], _dt(case), lo)
    for _ in range(steps):
        pos, vel, p, n = flow.step(type_, pos, vel, p, n, scene)
    out = dict(zip(axes, pos)) | dict(zip(vels, vel)) | {"p": p, "n": n, "type": None}
    return out


def _permutations(n, epochs):
    """The trainer's seeded Fisher-Yates shuffles (SplitMix64 from seed 0), one per epoch."""
    mask = (1 << 64) - 1
    state, out = 0, []
    for _ in range(epochs):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        out.append(torch.tensor(perm, device="cuda"))
    return out


def _exact_train(case, seed):
    blob, smp = _samples(case, seed)
    blob, smp = torch.from_numpy(blob).double().cuda(), torch.from_numpy(smp).double().cuda()
    mu, sd = blob[:16], blob[16:32]
    w = blob[32:].clone().requires_grad_(True)
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    shapes = [(64, 16), (64,), (64, 64), (64,), (64, 64), (64,), (2, 64), (2,)]
    sizes = [math.prod(s) for s in shapes]
    step, losses = 0, []
    bsz = min(case["batch"], case["n"])
    for perm in _permutations(case["n"], case["epochs"]):
        total = 0.0
        for at in range(0, case["n"], bsz):
            s = smp[perm[at:at + bsz]]
            P = [t.reshape(q) for t, q in zip(torch.split(w, sizes), shapes)]
            h = (s[:, :16] - mu) / sd
            for k in range(3):
                h = torch.nn.functional.gelu(h @ P[2 * k].T + P[2 * k + 1])
            o = h @ P[6].T + P[7]
            y, g = s[:, 16], s[:, 17]
            loss = ((o[:, 0] - y) ** 2 + (y - (1 + 0.25 * torch.tanh(o[:, 1])) * g) ** 2).sum()
            (grad,) = torch.autograd.grad(loss / s.shape[0], w)
            total += float(loss.detach())
            step += 1
            with torch.no_grad():
                m = 0.9 * m + 0.1 * grad
                v = 0.999 * v + 0.001 * grad * grad
                w -= 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        losses.append(total / case["n"])
    return {"blob": torch.cat([blob[:32], w.detach()]), "loss": torch.tensor(losses, dtype=torch.float64)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step2":
        s = _scene2(case, seed)
        return _exact_flow(case, [s], 2, (s.min_x, s.min_z), 1)
    if kind == "step3":
        s = _scene3(case, seed)
        return _exact_flow(case, [s], 3, s.bounds[:3], 1)
    if kind == "batch":
        parts = _batch_scenes(case, seed)
        return _exact_flow(case, parts, 2, (parts[0].min_x, parts[0].min_z), case["steps"])
    if kind == "csr":
        ptr, col, val, b = _csr(case, seed)
        n = b.numel()
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), ptr[1:] - ptr[:-1])
        off = row != col
        return _solve(row[off], col[off].long(), val[off], val[~off], b, torch.zeros_like(b))
    return _exact_train(case, seed)
