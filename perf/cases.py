"""Performance cases: what a simulation program has this library do.

Three kinds of program use it, and each case is one of theirs:

  system   one simulation: roll a stored state forward by some steps
           (ParticleSystem: WCSPH, PCISPH, rigid and granular coupling);
  batch    many independent scenes advanced together, the states read back
           to the host as a learning loop does (ParticleBatch);
  adjoint  the loss of a trajectory and its gradient (Adjoint).

A pass of the first two restores a checkpoint and steps, so that every pass
does the same work. `settle` steps (part of the preparation) take a scene out
of its start-up transient, in which the predict-correct loop runs to its cap;
`tuned` scenes keep the launch shapes that the library's autotuner picks, the
others its defaults. Seeds move the jitter of the lattices,
never the sizes.
"""
from __future__ import annotations

import ctypes as C
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import unifiedparticleframeworkcuda_b200 as upf
from unifiedparticleframeworkcuda_b200 import scenes

# the largest sizes drawn: those of the largest listed cases
MAX_WCSPH_SIDE, MAX_PCISPH, MAX_BATCH_SCENES, MAX_BATCH_COUNT = 61, 1 << 20, 256, 65536
MAX_ADJOINT_WORK = 65536 * 200
TERMS = upf.FLAG_SURFACE_TENSION | upf.FLAG_PENALTY_WALLS | upf.FLAG_BOUNDARY_PRESSURE | upf.FLAG_ADHESION


def listed():
    return [
        # the smallest scenes of the test suite (1,728 particles): interactive
        # previews, where launches and latency are everything
        {"name": "wcsph_2k", "kind": "wcsph", "side": 12, "terms": False, "steps": 4},
        {"name": "pcisph_2k", "kind": "pcisph", "nx": 12, "ny": 12, "nz": 12, "terms": False, "settle": 0,
         "tuned": False, "steps": 1},
        # the WCSPH dam break of the benchmark, 32,768 particles
        {"name": "wcsph_32k", "kind": "wcsph", "side": 32, "terms": False, "steps": 1},
        # a ragged scene of middle size with every optional PCISPH term, from rest
        {"name": "pcisph_53k_terms", "kind": "pcisph", "nx": 47, "ny": 39, "nz": 29, "terms": True, "settle": 0,
         "tuned": False, "steps": 1},
        # the largest WCSPH scene its grid holds, odd side, wall weight and surface tension
        {"name": "wcsph_227k_terms", "kind": "wcsph", "side": 61, "terms": True, "steps": 1},
        # a PCISPH dam at the size the profiles use, default launch shapes, settled
        {"name": "pcisph_262k", "kind": "pcisph", "nx": 64, "ny": 64, "nz": 64, "terms": False, "settle": 50,
         "tuned": False, "steps": 2},
        # the headline dam break: 1,048,576 particles, settled and tuned
        {"name": "pcisph_1m", "kind": "pcisph", "nx": 128, "ny": 128, "nz": 64, "terms": False, "settle": 50,
         "tuned": True, "steps": 2},
        # rigid bodies and a granular pile in a fluid, 748,431 dynamic particles
        {"name": "coupling_524k", "kind": "coupling", "nx": 128, "ny": 64, "nz": 64, "bodies": 16, "settle": 20,
         "tuned": True, "steps": 1},
        # a few uneven scenes at once, default launch shapes
        {"name": "batch_12", "kind": "batch", "scenes": 12, "lo": 2048, "hi": 16384, "settle": 0, "tuned": False,
         "steps": 1},
        # the benchmark's batch: 256 scenes, 5.2 million particles
        {"name": "batch_256", "kind": "batch", "scenes": 256, "lo": 2048, "hi": 65536, "settle": 5, "tuned": True,
         "steps": 2},
        # gradients of a short and of the benchmark's trajectory
        {"name": "adjoint_4k", "kind": "adjoint", "nx": 16, "ny": 16, "nz": 16, "steps": 20, "interval": 20,
         "loops": 3},
        {"name": "adjoint_65k", "kind": "adjoint", "nx": 32, "ny": 32, "nz": 64, "steps": 200, "interval": 20,
         "loops": 3},
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, lo, hi):
    """Three odd or even edges of a block of about lo..hi particles, none over 128."""
    n = _log_between(rng, lo, hi)
    a = max(4, min(128, int(round(n ** (1 / 3) * rng.uniform(0.7, 1.5)))))
    b = max(4, min(128, int(round(math.sqrt(n / a) * rng.uniform(0.8, 1.25)))))
    c = max(4, min(64, n // (a * b)))
    return a, b, c


def draw(rng):
    kind = rng.choice(["wcsph", "wcsph", "pcisph", "pcisph", "pcisph", "coupling", "batch", "batch", "adjoint"])
    if kind == "wcsph":
        return {"kind": kind, "side": _log_between(rng, 8, MAX_WCSPH_SIDE), "terms": rng.random() < 0.5,
                "steps": rng.choice([1, 2, 4])}
    if kind == "pcisph":
        nx, ny, nz = _block(rng, 1000, MAX_PCISPH)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "terms": rng.random() < 0.4,
                "settle": rng.choice([0, 25, 50]), "tuned": rng.random() < 0.3, "steps": rng.choice([1, 2])}
    if kind == "coupling":
        nx, ny, nz = _block(rng, 30000, 524288)
        nx, ny, nz = max(nx, 32), min(max(ny, 12), 64), max(nz, 32)
        # the bodies, up to 0.3 m across, stand side by side over the fluid
        across = int(0.01 * min(1.5 * nx + 8, 2 * nz + 2) / 0.32)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "bodies": rng.randint(1, min(16, across ** 2)),
                "settle": rng.choice([0, 20]), "tuned": rng.random() < 0.3, "steps": 1}
    if kind == "batch":
        hi = _log_between(rng, 2048, MAX_BATCH_COUNT)
        return {"kind": kind, "scenes": _log_between(rng, 2, MAX_BATCH_SCENES), "lo": max(500, hi // 16), "hi": hi,
                "settle": rng.choice([0, 5]), "tuned": rng.random() < 0.3, "steps": rng.choice([1, 2])}
    nx, ny, nz = _block(rng, 1000, 65536)
    steps = max(2, min(200, _log_between(rng, 5, 200), MAX_ADJOINT_WORK // (nx * ny * nz)))
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "interval": rng.choice([5, 10, 20]),
            "loops": rng.choice([1, 2, 3])}


# ---------------------------------------------------------------- scenes
def _scene(case, seed):
    kind = case["kind"]
    if kind == "wcsph":
        side = case["side"]
        # the container of the benchmark's dam (1 m for 32), scaled
        sc = scenes.wcsph_dam(side, seed=seed, box=0.02 * max(20, min(68, math.ceil(1.56 * side))))
        sc.params.dt = 5e-4  # 0.4 h / c, the sound-speed limit of this stiffness
        if case["terms"]:
            sc.params.flags = upf.FLAG_WALL_WEIGHT | upf.FLAG_SURFACE_TENSION
        return sc
    if kind == "pcisph":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s = 0.01
        box = (s * min(200, math.ceil(1.5625 * nx)), s * (ny + 2), s * (2 * nz + 2))
        sc = scenes.pcisph_dam(nx, ny, nz, seed=seed, box=box, spacing=s)
        if case["terms"]:
            sc.params.flags = TERMS
            sc.params.surface_adhesion_beta = 0.5
        return sc
    if kind == "coupling":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        grains = (max(4, nx // 2), max(2, ny // 2), nz)
        s = 0.01
        box = (s * min(200, nx + grains[0] + 8), s * (ny + 66), s * min(196, 2 * nz + 2))
        sc = scenes.coupling_scene((nx, ny, nz), grains, n_bodies=case["bodies"], box=box)
        # the same bodies for every seed, which moves the fluid and the grains
        loose = (sc.type == upf.LIQUID) | (sc.type == upf.GRANULAR)
        sc.pos[loose, :3] += (scenes.uniform(seed, 3 * sc.n).reshape(sc.n, 3)[loose] - 0.5) * (0.1 * s)
        return sc
    if kind == "adjoint":
        return scenes.adjoint_scene(case["nx"], case["ny"], case["nz"], seed=seed)
    raise ValueError("unknown kind %r" % (kind,))


_derived = {}


def _batch_scenes(case, seed):
    """The batch's scenes: counts and boxes from the case, jitter from the seed."""
    num = case["scenes"]
    u = scenes.uniform(2024, 4 * num, stream=7).reshape(num, 4)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])

    def make(k):
        n = int(round(math.exp(lo + (hi - lo) * u[k, 0])))
        return scenes.batch_scene(n, 0.5 + 1.5 * u[k, 1:4], seed + 17 * k, stream=k + 1)

    with ThreadPoolExecutor(8) as ex:
        scs = list(ex.map(make, range(num)))
        key = (num, case["lo"], case["hi"])
        if key not in _derived:  # a program derives its scenes' parameters once
            _derived[key] = list(ex.map(lambda sc: upf.derive_params(sc.params), scs))
    return scs, _derived[key]


def _params(case, sc):
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "settle", "tuned", "interval")))
    if key not in _derived:
        _derived[key] = upf.derive_params(sc.params)
    return _derived[key]


_stream = None


def _program_stream():
    """The one stream the program runs its simulations on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


class _View:
    """A device array of a system, seen by torch without a copy (CUDA array
    interface); it keeps the system, whose memory it is."""

    def __init__(self, system, ptr, shape, typestr):
        self.system = system
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "version": 3, "strides": None,
                                         "data": (C.cast(ptr, C.c_void_p).value, False)}


def prepare(case, seed):
    if case["kind"] == "batch":
        scs, params = _batch_scenes(case, seed)
        b = upf.ParticleBatch(params, [sc.n for sc in scs], derive=False)
        b.set_stream(_program_stream())
        b.set_particles(np.concatenate([sc.pos for sc in scs]), np.concatenate([sc.vel for sc in scs]))
        if case["settle"]:
            b.step(case["settle"])
        if case["tuned"]:
            b.autotune(3)
        b.checkpoint(0)
        b.synchronize()
        n = int(b.offsets[-1])
        pos, vel = (torch.empty((n, 4), dtype=torch.float32, pin_memory=True) for _ in range(2))
        return {"batch": b, "steps": case["steps"], "pos": pos, "vel": vel}
    sc = _scene(case, seed)
    params = _params(case, sc)
    if case["kind"] == "adjoint":
        a = upf.Adjoint(params, sc.pos, sc.vel, steps=case["steps"], checkpoint_interval=case["interval"],
                        loop_iterations=case["loops"], target=_TARGET, density_weight=_DENSITY_WEIGHT, derive=False)
        a.set_stream(_program_stream())
        return {"adjoint": a, "vel": sc.vel}
    s = upf.ParticleSystem(params, capacity=sc.n, derive=False)
    s.set_stream(_program_stream())
    s.set_particles(sc.pos, sc.vel, sc.type)
    if sc.num_bodies:
        s.set_rigid_bodies(sc.body, sc.num_bodies)
    if case.get("settle"):
        s.step(case["settle"])
    if case.get("tuned"):
        s.autotune(3)
    s.checkpoint(0)
    s.synchronize()
    # the state's device arrays, as a program that renders or learns on the GPU reads them
    d = upf.UpfDeviceState()
    upf.check(upf.lib().upf_get_device_state(s.handle, C.byref(d)), "upf_get_device_state")

    def view(ptr, cols, typestr="<f4"):
        return torch.as_tensor(_View(s, ptr, (d.n, cols) if cols else (d.n,), typestr), device="cuda")

    out = {"pos": view(d.pos4, 4), "vel": view(d.vel4, 4), "id": view(d.id, 0, "<i4"),
           "density": view(d.density, 0), "pressure": view(d.pressure, 0)}
    if case["kind"] != "wcsph":
        out["lag"] = view(d.lag4, 4)
    if case["kind"] == "coupling":
        # density and pressure are the liquid's: the solids' entries are not written by a step
        del out["density"], out["pressure"]
    return {"system": s, "steps": case["steps"], "out": out}


def run(state):
    if "system" in state:
        s = state["system"]
        s.restore(0)
        s.step(state["steps"])
        return state["out"]
    if "batch" in state:
        b = state["batch"]
        b.restore(0)
        b.step(state["steps"])
        fp = C.POINTER(C.c_float)
        upf.check(upf.lib().upf_batch_download_state(b.handle, C.cast(state["pos"].data_ptr(), fp),
                                                     C.cast(state["vel"].data_ptr(), fp)), "upf_batch_download_state")
        return {"pos": state["pos"], "vel": state["vel"]}
    a = state["adjoint"]
    loss = a.forward(state["vel"])
    grad_vel, grad_viscosity = a.backward()
    pos, vel = a.state()
    return {"loss": loss, "grad_vel": grad_vel, "grad_viscosity": grad_viscosity, "pos": pos, "vel": vel}


# ---------------------------------------------------------------- work
NEIGHBORS = 30  # within h = 2 spacings of a lattice particle, about


def work(case):
    """Bytes: a step's state read and written once (position, velocity, type,
    id; the lagged pressures of PCISPH), the boundary read once. Operations:
    per neighbour 8 for its distance, then 2 (density), 16 (pressure force)
    and 25 (viscosity, surface tension) per pass; the loop's iterations at
    what such scenes take (the cap from rest, 14 settled)."""
    kind = case["kind"]
    if kind == "adjoint":
        n, steps, k = case["nx"] * case["ny"] * case["nz"], case["steps"], case["loops"]
        per_step = NEIGHBORS * (8 * (1 + 2 * k) + 10 + k * (2 + 12))
        # forward, the forward again from checkpoints, and the adjoint at twice the forward's operations
        return {"bytes": 4.0 * n * 16 * 3, "flops": float(n) * steps * per_step * 4}
    if kind == "batch":
        num = case["scenes"]
        u = scenes.uniform(2024, 4 * num, stream=7).reshape(num, 4)[:, 0]
        n = float(np.sum(np.exp(math.log(case["lo"]) + (math.log(case["hi"]) - math.log(case["lo"])) * u)))
        state, wall, k = 56, 0.0, 6
    elif kind == "wcsph":
        n, state = float(case["side"]) ** 3, 40
        wall, k = 16.0 * 6 * (1.56 * case["side"]) ** 2, 0
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n, state = float(nx * ny * nz), 56
        wall = 16.0 * 2 * 2 * (1.56 * nx * ny + 2 * 1.56 * nx * nz + 2 * ny * nz)
        k = 14 if case["settle"] else 50
        if kind == "coupling":
            n, k = n * 1.4, 35
    per = NEIGHBORS * ((8 + 25) + k * (8 + 2 + 16)) if k else NEIGHBORS * (8 + 2 + 16 + 25)
    return {"bytes": case["steps"] * (2.0 * state * n + wall), "flops": case["steps"] * n * per}


# ---------------------------------------------------------------- 64 bits
# The methods in double precision on torch, for the outputs' error: the
# 300-bin kernel tables (evaluated in double at the bins' lower edges), the
# neighbours found by a uniform grid, the Morton order of the outputs from
# the single-precision keys.
_TARGET, _DENSITY_WEIGHT = (1.0, 1.0, 1.0), 1e-6
BINS = 300


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        # longer trajectories take minutes in 64 bits
        if case["nx"] * case["ny"] * case["nz"] * case["steps"] * case["loops"] > 300_000:
            return None
        sc = _scene(case, seed)
        return _exact_adjoint(case, _params(case, sc), sc)
    if case.get("settle") or kind == "coupling":
        # a settled state is the library's own: from the seed alone it is tens of
        # steps at the iteration cap, minutes in 64 bits
        return None
    if kind == "batch":
        scs, params = _batch_scenes(case, seed)
        if sum(sc.n for sc in scs) * case["steps"] > 200_000:
            return None
        outs = [_Exact(p, sc).steps(case["steps"]) for sc, p in zip(scs, params)]
        return {k: torch.cat([o[k] for o in outs]).cpu() for k in ("pos", "vel")}
    sc = _scene(case, seed)
    if kind == "pcisph" and sc.n_fluid * case["steps"] > 200_000:
        return None
    out = _Exact(_params(case, sc), sc).steps(case["steps"])
    if kind == "wcsph":
        del out["lag"]
    return out


def _pairs(x, y, h):
    """(i, j) with |x_i - y_j| < h."""
    lo = torch.minimum(x.min(0).values, y.min(0).values) - 1e-9
    side = int(((torch.maximum(x.max(0).values, y.max(0).values) - lo) / h).max().item()) + 3
    cell = lambda p: (((p - lo) / h).long() + 1)  # noqa: E731
    flat = lambda c: (c[:, 0] * side + c[:, 1]) * side + c[:, 2]  # noqa: E731
    key, order = torch.sort(flat(cell(y)))
    cx = cell(x)
    out_i, out_j = [], []
    rows = torch.arange(x.shape[0], device=x.device)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            want = flat(cx + torch.tensor([dx, dy, 0], device=x.device))
            # the three cells along z follow one another
            b, e = torch.searchsorted(key, want - 1), torch.searchsorted(key, want + 1, right=True)
            cnt = e - b
            i = torch.repeat_interleave(rows, cnt)
            first = torch.repeat_interleave(b - (torch.cumsum(cnt, 0) - cnt), cnt)
            j = order[first + torch.arange(i.shape[0], device=x.device)]
            near = ((x[i] - y[j]) ** 2).sum(1) < h * h
            out_i.append(i[near])
            out_j.append(j[near])
    return torch.cat(out_i), torch.cat(out_j)


def _sum_at(i, v, n):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add_(0, i, v)


def _m4(r, h):
    s = r / h
    return 8 / (math.pi * h ** 3) * torch.where(s < 0.5, 1 - 6 * s ** 2 + 6 * s ** 3,
                                                2 * (1 - s).clamp(min=0) ** 3)


def _cohesion(r, h):
    near = 2 * (h - r) ** 3 * r ** 3 - h ** 6 / 64
    v = torch.where(r > 0.5 * h, (h - r) ** 3 * r ** 3, near)
    return 32 / (math.pi * h ** 9) * torch.where(r > 0, v, torch.zeros_like(v))


class _Exact:
    """A liquid in a frozen boundary, in double precision."""

    def __init__(self, p, sc):
        self.p = p
        dev = torch.device("cuda", 0)
        f64 = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        liquid = sc.type == upf.LIQUID
        self.x, self.v, self.xb = f64(sc.pos[liquid, :3]), f64(sc.vel[liquid, :3]), f64(sc.pos[~liquid, :3])
        self.ids = torch.tensor(np.nonzero(liquid)[0].astype(np.int32), device=dev)
        n = self.x.shape[0]
        self.lag = torch.zeros((n, 4), dtype=torch.float64, device=dev)
        self.lag[:, 2] = p.rest_density
        self.h = h = float(p.support_radius)
        r = torch.arange(BINS, dtype=torch.float64, device=dev) * (h / BINS)
        zero = torch.zeros(1, dtype=torch.float64, device=dev)
        c = 45 / (math.pi * h ** 6)
        grad = -c * (h - r) ** 2 / r
        grad[0] = 0
        base = (-4 * r * r / h + 6 * r - 2 * h).clamp(min=0)
        adhesion = torch.where(r > 0.5 * h, 0.007 / h ** 3.25 * base ** 0.25, torch.zeros_like(r))
        self.t_m4, self.t_grad, self.t_lap, self.t_coh, self.t_adh = (
            torch.cat([t, zero]) for t in (_m4(r, h), grad, c * (h - r), _cohesion(r, h), adhesion))
        self.w0 = 8 / (math.pi * h ** 3)
        self.lo, self.hi = f64(p.collision_min[:]), f64(p.collision_max[:])
        self.m, self.rho0 = float(p.mass), float(p.rest_density)
        self.down = f64([0.0, self.m * p.gravity, 0.0])
        # volumes of the boundary particles
        i, j = _pairs(self.xb, self.xb, h) if len(self.xb) else (None, None)
        if i is not None:
            i, j = i[i != j], j[i != j]
            w = _sum_at(i, self.t_m4[self._bin((self.xb[i] - self.xb[j]).norm(dim=1))], len(self.xb))
            self.vol_b = torch.where(w > 0, 1 / w, torch.full_like(w, self.m / self.rho0))

    def _bin(self, d):
        return (d * (BINS / self.h)).long().clamp(max=BINS)

    def steps(self, count):
        for _ in range(count):
            rho, press = self._step()
        pad = torch.zeros((len(self.x), 1), dtype=torch.float64, device=self.x.device)
        return {"pos": torch.cat([self.x, pad], 1), "vel": torch.cat([self.v, pad], 1), "id": None,
                "density": rho, "pressure": press, "lag": self.lag}

    def _sort(self):
        p = self.p
        x = self.x.float().cpu().numpy()
        c = (np.array(p.scales[:], np.float32) * (x - np.array(p.zindex_origin[:], np.float32)))
        c = np.clip(c, 0, 1023).astype(np.int64)
        key = np.zeros(len(x), np.int64)
        for b in range(10):
            for a in range(3):
                key |= ((c[:, a] >> b) & 1) << (3 * b + a)
        at = torch.tensor(np.argsort(key, kind="stable"), device=self.x.device)
        self.x, self.v, self.lag = self.x[at], self.v[at], self.lag[at]

    def _neighbors(self):
        x, n = self.x, len(self.x)
        i, j = _pairs(x, x, self.h)
        i, j = i[i != j], j[i != j]
        d = (x[i] - x[j]).norm(dim=1)
        if not len(self.xb):
            return (i, j, d), (i[:0], j[:0], d[:0])
        bi, bj = _pairs(x, self.xb, self.h)
        return (i, j, d), (bi, bj, (x[bi] - self.xb[bj]).norm(dim=1))

    def _step(self):
        self._sort()
        return self._wcsph() if self.p.method == upf.METHOD_WCSPH else self._pcisph()

    def _integrate(self, f):
        self.v = self.v + f * (self.p.dt / self.m)
        self.x = self.x + self.v * self.p.dt
        out = (self.x < self.lo) | (self.x > self.hi)
        self.x = torch.minimum(torch.maximum(self.x, self.lo), self.hi)
        self.v = torch.where(out, -0.5 * self.v, self.v)

    def _cohere(self, dx, d, strength, table):
        """Surface tension or adhesion of pairs, per unit of `strength`."""
        return torch.where((d >= 0.25 * self.h)[:, None], dx * (strength * table / d)[:, None], torch.zeros_like(dx))

    def _wcsph(self):
        p, n, m = self.p, len(self.x), self.m
        (i, j, d), (bi, _, bd) = self._neighbors()
        b = self._bin(d)
        rho = self.w0 * m + m * (_sum_at(i, self.t_m4[b], n) + _sum_at(bi, self.t_m4[self._bin(bd)], n))
        if p.flags & upf.FLAG_WALL_WEIGHT:
            rho = rho + self._wall_weight()
        gas = self.rho0 * p.gas_constant / p.gamma
        press = (gas * ((rho / self.rho0) ** p.gamma - 1)).clamp(min=0)
        dx = self.x[i] - self.x[j]
        q = press / rho ** 2
        f = -dx * (self.t_grad[b] * (q[i] + q[j]) * m * m)[:, None]
        f = f - (self.v[i] - self.v[j]) * (p.viscosity * self.t_lap[b] * (m / rho[i]) * (m / rho[j]))[:, None]
        if p.flags & upf.FLAG_SURFACE_TENSION:
            f = f - self._cohere(dx, d, p.surface_tension_gamma * m * m, _cohesion(d, self.h))
        self._integrate(_sum_at(i, f, n) - self.down)
        return rho, press

    def _wall_weight(self):
        p, r, s = self.p, float(self.p.particle_radius), float(self.p.particle_spacing)
        lo, hi = (torch.tensor(np.array(a[:], np.float64), device=self.x.device)
                  for a in (p.container_min, p.container_max))
        near = torch.minimum((self.x - lo).clamp(min=0), (hi - self.x).clamp(min=0)).min(1).values
        near = near.clamp(max=float((hi - lo).max()))
        w = lambda d: self.t_m4[self._bin(d)]  # noqa: E731
        d1 = near + r
        d2 = d1 + s
        side = lambda d, k: (d * d + (k * s) ** 2).sqrt()  # noqa: E731
        total = w(d1) + w(d2) + 2 * (w(side(d1, 1)) + w(side(d1, 2)) + w(side(d2, 1)) + w(side(d2, 2)))
        return torch.where(near >= self.h - r, torch.zeros_like(total), self.m * total)

    def _pcisph(self):
        p, n, m = self.p, len(self.x), self.m
        (i, j, d), (bi, bj, bd) = self._neighbors()
        b, vol = self._bin(d), m / self.rho0
        dx = self.x[i] - self.x[j]
        f = -(self.v[i] - self.v[j]) * (vol * vol * p.viscosity * self.t_lap[b])[:, None]
        if p.flags & upf.FLAG_SURFACE_TENSION:
            f = f - self._cohere(dx, d, p.surface_tension_gamma * m * m, self.t_coh[b])
        force = _sum_at(i, f, n) - self.down
        if len(bi):
            bb, bdx = self._bin(bd), self.x[bi] - self.xb[bj]
            fb = torch.zeros_like(bdx)
            if p.flags & upf.FLAG_BOUNDARY_PRESSURE:
                lagged = self.lag[:, 0] / self.lag[:, 2] ** 2
                fb = fb - bdx * (self.t_grad[bb] * lagged[bi] * m * self.rho0 * vol)[:, None]
            if p.flags & upf.FLAG_ADHESION:
                fb = fb - self._cohere(bdx, bd, p.surface_adhesion_beta * m * self.rho0 * self.vol_b[bj],
                                       self.t_adh[bb])
            force = force + _sum_at(bi, fb, n)
        if p.flags & upf.FLAG_PENALTY_WALLS:
            fd = float(p.force_distance)
            k = 2 * float(p.max_boundary_force) / fd
            force = force + k * ((self.lo + fd - self.x).clamp(min=0) - (self.x + fd - self.hi).clamp(min=0))
        press = torch.zeros(n, dtype=torch.float64, device=self.x.device)
        fp = torch.zeros_like(force)
        # all neighbours, the boundary's behind the liquid's: fixed, and without pressure
        ai, aj = torch.cat([i, bi]), torch.cat([j, bj + n])
        adx = torch.cat([dx, self.x[bi] - self.xb[bj]])
        grad = self.t_grad[self._bin(torch.cat([d, bd]))]
        too_large, it = True, 0
        while True:
            xs = self.x + (self.v + (force + fp) * (p.dt / m)) * p.dt
            xs = torch.minimum(torch.maximum(xs, self.lo), self.hi)
            far = torch.cat([xs, self.xb])
            rho = self.w0 * m + m * _sum_at(ai, self.t_m4[self._bin((xs[ai] - far[aj]).norm(dim=1))], n)
            press = press + p.density_error_factor * (rho - self.rho0).clamp(min=0)
            q = torch.cat([press / self.rho0 ** 2, torch.zeros(len(self.xb), dtype=torch.float64, device=xs.device)])
            fp = _sum_at(ai, -adx * (grad * (q[ai] + q[aj]) * m * m)[:, None], n)
            it += 1
            if max(100 / self.rho0 * float(rho.max()) - 100, 0) < p.max_density_error:
                too_large = False
            if not (it < p.min_loops or (too_large and it < p.max_loops)):
                break
        self.lag = torch.stack([self.lag[:, 1], press, rho, torch.zeros_like(rho)], 1)
        self._integrate(force + fp)
        return rho, press


def _exact_adjoint(case, p, sc):
    """The smoothed trajectory and its gradient by automatic differentiation."""
    dev = torch.device("cuda", 0)
    f64 = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    h, m, rho0, dt = float(p.support_radius), float(p.mass), float(p.rest_density), float(p.dt)
    vol, eps, c = m / rho0, 0.01 * rho0, 45 / (math.pi * h ** 6)
    lo, hi = f64(p.collision_min[:]), f64(p.collision_max[:])
    down = f64([0.0, m * p.gravity, 0.0])
    v0 = f64(sc.vel[:, :3]).requires_grad_()
    mu = torch.tensor(float(p.viscosity), dtype=torch.float64, device=dev, requires_grad=True)
    x, v, n = f64(sc.pos[:, :3]), v0, sc.n

    def dist(a, i, j):
        return ((a[i] - a[j]) ** 2).sum(1).sqrt()

    def density(a, i, j):
        r = dist(a, i, j)
        return m * _m4(torch.zeros((), dtype=torch.float64, device=dev), h) + m * _sum_at(
            i, torch.where(r < h, _m4(r, h), torch.zeros_like(r)), n)

    def near(a):
        i, j = _pairs(a.detach(), a.detach(), h)
        return i[i != j], j[i != j]

    for _ in range(case["steps"]):
        i, j = near(x)
        d = dist(x, i, j)
        force = _sum_at(i, -(v[i] - v[j]) * (vol * vol * mu * c * (h - d))[:, None], n) - down
        fp, press = torch.zeros_like(force), torch.zeros(n, dtype=torch.float64, device=dev)
        grad = (x[i] - x[j]) * (-c * (h - d) ** 2 / d)[:, None]
        for _ in range(case["loops"]):
            xs = x + (v + (force + fp) * (dt / m)) * dt
            xs = torch.minimum(torch.maximum(xs, lo), hi)
            e = density(xs, i, j) - rho0
            press = press + p.density_error_factor * 0.5 * (e + (e * e + eps * eps).sqrt())
            fp = _sum_at(i, -grad * (m * m / rho0 ** 2 * (press[i] + press[j]))[:, None], n)
        v = v + (force + fp) * (dt / m)
        x = x + v * dt
    i, j = near(x)
    loss = ((x.mean(0) - f64(_TARGET)) ** 2).sum() + _DENSITY_WEIGHT * ((density(x, i, j) - rho0) ** 2).mean()
    g_v, g_mu = torch.autograd.grad(loss, [v0, mu])
    pad = torch.zeros((n, 1), dtype=torch.float64, device=dev)
    return {"loss": float(loss), "grad_vel": g_v, "grad_viscosity": float(g_mu),
            "pos": torch.cat([x.detach(), pad], 1), "vel": torch.cat([v.detach(), pad], 1)}
