"""What the particle path's users have it do, as cases that can be prepared, run and timed.

Every case goes through the public entry points (``PicContext`` and the C ABI behind it).  The
kinds, and what each stands for:

``simulate``  a run between two outputs: the swarm is seeded, located, advanced a number of steps
              on the device, and the swarm, the scattered fields and the face deposits come back
              in the reference's DMSwarm / DMDA layouts in page-locked arrays.  ``monitor`` reads
              the step's counts after every step, as the reference's loop logs them.
``exchange``  a host code that owns the DMSwarm: velocity field and swarm up, one step, swarm and
              fields down.
``coupled``   a flow solver on the same GPU: the contravariant face velocity changes every step
              and is converted on the device before the particles move.
``points``    caller-held particles (a DMSwarm kept on the host, probes): their walk, then the
              velocity at them.
``sort``      the standalone sort by cell on device arrays.
``train``     the learned locator made for a new grid: training and a prediction with it.
``infer``     a locator whose weights are there: loss and gradients on a held-out batch, and a
              prediction.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fdf_gb300.context import FORM_FP32, FORM_LEARNED_FP32, FORM_PLAIN_FP64, LOCATOR_NPARAM, PicContext, SwarmArrays

FORMS = {"plain": FORM_PLAIN_FP64, "fp32": FORM_FP32, "learned": FORM_LEARNED_FP32}
DEV = "cuda"
F64 = torch.float64
ATMOSPHERE = 101325.0
VOLUME = 1.0e-6


def listed():
    return [
        # The smallest run anyone makes: the reference's own test box, every particle walked in
        # from the corner cell, counts logged after every step.
        dict(name="uniform_10k_plain", kind="simulate", grid="uniform", IM=20, JM=20, KM=280, n=10_000, cfl=0.1,
             steps=10, form="plain", corner=True, monitor=True, momentum=False),
        # An ordinary bit-exact run on a curvilinear box: fewer particles than cells.
        dict(name="sinusoidal_1m_plain", kind="simulate", grid="sinusoidal", IM=64, JM=64, KM=1024, n=1_000_000,
             cfl=0.5, steps=50, form="plain", corner=False, monitor=False, momentum=False),
        # An ordinary precision-form run; one particle in eighty sits in a gap between two cells' planes
        # and is LOST at the start.
        dict(name="sinusoidal_6m_fp32", kind="simulate", grid="sinusoidal", IM=96, JM=96, KM=1536, n=6_000_000,
             cfl=1.0, steps=20, form="fp32", corner=False, monitor=False, momentum=False),
        # The bit-exact form on a pipe bend, particles crossing several cells per step.
        dict(name="bent_pipe_16m_plain", kind="simulate", grid="bent_pipe", IM=96, JM=96, KM=1536, n=16_000_000,
             cfl=4.0, steps=8, form="plain", corner=False, monitor=False, momentum=False),
        # The largest: the learned form at the benchmark's size.
        dict(name="bent_pipe_64m_learned", kind="simulate", grid="bent_pipe", IM=96, JM=96, KM=1536, n=64_000_000,
             cfl=4.0, steps=20, form="learned", corner=False, monitor=False, momentum=False),
        # Volume and momentum handed back to a flow solver, four particles per cell, odd sizes.
        dict(name="curved_pipe_momentum", kind="simulate", grid="curved_pipe", IM=61, JM=67, KM=1021, n=15_999_937,
             cfl=1.0, steps=20, form="fp32", corner=False, monitor=False, momentum=True),
        # A PETSc host code's step with the swarm and the field on the host.
        dict(name="exchange_2m_plain", kind="exchange", grid="bent_pipe", IM=48, JM=48, KM=384, n=2_000_000, cfl=1.0,
             form="plain"),
        # A flow solver on the same GPU, its face velocity converted every step.
        dict(name="coupled_2m_fp32", kind="coupled", grid="sinusoidal", IM=64, JM=64, KM=512, n=2_000_000, cfl=1.0,
             steps=10, form="fp32"),
        # Caller-held particles: the walk and the interpolation of a host loop.
        dict(name="points_200k", kind="points", grid="sinusoidal", IM=64, JM=64, KM=512, n=200_000, hint=True),
        # The sort alone, on ids as a step leaves them (nearly in order, some particles gone).
        dict(name="sort_16m", kind="sort", n=16_000_000, ncells=4_000_037, spread=4096, gone=0.002),
        # A locator made for a new grid.
        dict(name="train_500", kind="train", grid="bent_pipe", IM=48, JM=48, KM=384, samples=1_000_000, steps=500,
             batch=8192, n=200_000),
        # A locator used and checked.
        dict(name="infer_500k", kind="infer", grid="bent_pipe", IM=48, JM=48, KM=384, batch=8192, n=500_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most):
    """A grid of a family, 12 to 96 cells across and up to `most` cells."""
    while True:
        d = dict(grid=rng.choice(["uniform", "sinusoidal", "bent_pipe", "curved_pipe"]), IM=_log(rng, 12, 96),
                 JM=_log(rng, 12, 96), KM=_log(rng, 64, 1536))
        # the waves of the sinusoidal box take two dozen cells to resolve, and not too flat ones
        coarse = d["grid"] == "sinusoidal" and not (min(d["IM"], d["JM"]) >= 24 and d["KM"] <= 12 * min(d["IM"], d["JM"]))
        if d["IM"] * d["JM"] * d["KM"] <= most and not coarse:
            return d


def _crowd(g):
    """The most particles a run puts on a grid: two dozen per cell, fewer where many start LOST."""
    return min(24 * g["IM"] * g["JM"] * g["KM"], 2_000_000 if g["grid"] == "sinusoidal" else 48_000_000)


def draw(rng):
    kind = rng.choice(["simulate"] * 6 + ["exchange", "coupled", "points", "sort", "train", "infer"])
    if kind == "simulate":
        form = rng.choice(["plain", "fp32", "learned"])
        g = _grid(rng, 14_200_000)
        n = _log(rng, 5_000, min(16_000_000 if form == "plain" else 48_000_000, _crowd(g)))
        return dict(kind=kind, **g, n=n, cfl=rng.choice([0.25, 0.5, 1.0, 2.0, 4.0]),
                    steps=rng.randint(5, 10 if n > 4_000_000 else 30), form=form, corner=False,
                    monitor=n < 200_000 and rng.random() < 0.5, momentum=rng.random() < 0.25)
    if kind == "exchange":
        g = _grid(rng, 4_200_000)
        return dict(kind=kind, **g, n=_log(rng, 10_000, min(3_900_000, _crowd(g))), cfl=rng.choice([0.5, 1.0, 2.0]),
                    form=rng.choice(["plain", "fp32"]))
    if kind == "coupled":
        g = _grid(rng, 4_200_000)
        return dict(kind=kind, **g, n=_log(rng, 20_000, min(8_000_000, _crowd(g))), cfl=rng.choice([0.5, 1.0, 2.0]),
                    steps=rng.randint(5, 15), form=rng.choice(["plain", "fp32"]))
    if kind == "points":
        g = _grid(rng, 4_200_000)
        return dict(kind=kind, **g, n=_log(rng, 1_000, 2_000_000), hint=g["KM"] > 400 or rng.random() < 0.7)
    if kind == "sort":
        ncells = _log(rng, 10_000, 14_000_000)
        return dict(kind=kind, n=_log(rng, 10_000, min(32_000_000, 24 * ncells)), ncells=ncells,
                    spread=rng.choice([64, 4096, 1 << 20]), gone=rng.choice([0.0, 0.002, 0.05]))
    if kind == "train":
        return dict(kind=kind, **_grid(rng, 4_200_000), samples=_log(rng, 100_000, 4_000_000), steps=rng.randint(100, 1000),
                    batch=rng.choice([1024, 4096, 5000, 8192, 16384]), n=_log(rng, 1_000, 1_000_000))
    return dict(kind=kind, **_grid(rng, 4_200_000), batch=_log(rng, 16, 32_768), n=_log(rng, 1_000, 2_000_000))


# ------------------------------------------------------------------ inputs

def _axis(m):
    return torch.arange(m + 1, dtype=F64, device=DEV) / m


def _nodes(case):
    """Node coordinates [KM+1][JM+1][IM+1][3] of the case's grid, on the GPU."""
    IM, JM, KM, two_pi = case["IM"], case["JM"], case["KM"], 2.0 * math.pi
    Z, Y, X = torch.meshgrid(_axis(KM), _axis(JM), _axis(IM), indexing="ij")
    if case["grid"] == "uniform":
        return torch.stack([X, Y, Z], -1)
    if case["grid"] == "sinusoidal":
        sx, sy, sz = torch.sin(two_pi * X), torch.sin(two_pi * Y), torch.sin(two_pi * Z)
        return torch.stack([X + 0.04 * sy * sz, Y + 0.04 * sz * sx, Z + 0.04 * sx * sy], -1)
    # an O-type disk of radius 0.5 swept along a curve
    a, b = 2.0 * X - 1.0, 2.0 * Y - 1.0
    u, v = 0.5 * a * torch.sqrt(1.0 - 0.5 * b * b), 0.5 * b * torch.sqrt(1.0 - 0.5 * a * a)
    if case["grid"] == "bent_pipe":   # a quarter turn of radius 3: i inward, j up, k along the bend
        t = 0.5 * math.pi * Z
        g = torch.stack([(3.0 + u) * torch.cos(t), (3.0 + u) * torch.sin(t), v], -1)
        return torch.flip(g, [2]).contiguous()
    s = 8.0 * Z
    cx, d = torch.sin(math.pi * s / 8.0), (math.pi / 8.0) * torch.cos(math.pi * s / 8.0)
    t = torch.sqrt(1.0 + d * d)
    return torch.stack([cx + u / t, v, s - u * d / t], -1)


def _centres(x):
    return (x[:-1, :-1, :-1] + x[:-1, :-1, 1:] + x[:-1, 1:, :-1] + x[:-1, 1:, 1:] + x[1:, :-1, :-1] + x[1:, :-1, 1:]
            + x[1:, 1:, :-1] + x[1:, 1:, 1:]) / 8.0


def _velocity(case, x):
    """Cell-centred velocity [KM][JM][IM][3]: mostly along k, with swirl across."""
    c, two_pi = _centres(x), 2.0 * math.pi
    if case["grid"] in ("uniform", "sinusoidal"):
        if case["grid"] == "uniform":
            w = [0.1 * torch.sin(two_pi * c[..., 1]), 0.1 * torch.sin(two_pi * c[..., 2]),
                 1.0 + 0.1 * torch.sin(two_pi * c[..., 0])]
        else:
            w = [torch.sin(two_pi * c[..., 0]) * torch.cos(two_pi * c[..., 1]),
                 -torch.cos(two_pi * c[..., 0]) * torch.sin(two_pi * c[..., 1]), torch.ones_like(c[..., 0])]
        return torch.stack(w, -1)
    JM, IM = case["JM"], case["IM"]
    ctr = 0.5 * (x[:, JM // 2, IM // 2] + x[:, (JM + 1) // 2, (IM + 1) // 2])
    tang = ctr[1:] - ctr[:-1]
    tang = (tang / tang.norm(dim=-1, keepdim=True))[:, None, None, :]
    rel = c - (0.5 * (ctr[:-1] + ctr[1:]))[:, None, None, :]
    rel = rel - (rel * tang).sum(-1, keepdim=True) * tang
    r2 = (rel * rel).sum(-1, keepdim=True)
    axial = 2.0 * (1.0 - 4.0 * r2).clamp(min=0.0) * tang
    if case["grid"] == "bent_pipe":
        return axial
    swirl = torch.linalg.cross(tang.expand_as(rel), rel)
    return axial + 0.4 * torch.sin(two_pi * torch.sqrt(r2)) * swirl


def _dt(case, x, u):
    edge = min(float(torch.diff(x, dim=d).norm(dim=-1).min()) for d in range(3))
    return case.get("cfl", 1.0) * edge / float(u.norm(dim=-1).max())


def _lsr(z, s):
    return (z >> s) & ((1 << (64 - s)) - 1)


def _signed(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _mix(z):
    z = (z ^ _lsr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _lsr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _lsr(z, 31)


def _uniform01(seed, stream, n):
    """The first n doubles in [0, 1) of the splitmix64 stream that the seeding documents."""
    z = (seed * 0xD1B54A32D192ED03 + stream * 0xA24BAED4963EE407 + 0x632BE59BD9B4E019) & ((1 << 64) - 1)
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & ((1 << 64) - 1)
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & ((1 << 64) - 1)
    base = _signed(z ^ (z >> 31))
    idx = torch.arange(1, n + 1, dtype=torch.int64, device=DEV)
    return _lsr(_mix(base + idx * _signed(0x9E3779B97F4A7C15)), 11).to(F64) * (1.0 / 9007199254740992.0)


def _particles(case, x, n, seed):
    """n points of the volumetric initialisation: a random cell, random logical coordinates.
    Returns positions [n][3] and cells [n][3] (i, j, k)."""
    dims = (case["IM"], case["JM"], case["KM"])
    cell = [(_uniform01(seed, d, n) * dims[d]).to(torch.int64).clamp_(0, dims[d] - 1) for d in range(3)]
    lc = [_uniform01(seed, 3 + d, n).clamp_(0.0, 1.0 - 1.0e-7) for d in range(3)]
    flat, mx, my = x.reshape(-1, 3), case["IM"] + 1, case["JM"] + 1
    p = torch.zeros(n, 3, dtype=F64, device=DEV)
    for c in range(8):
        b = (c & 1, (c >> 1) & 1, (c >> 2) & 1)
        w = [lc[d] if b[d] else 1.0 - lc[d] for d in range(3)]
        node = ((cell[2] + b[2]) * my + cell[1] + b[1]) * mx + cell[0] + b[0]
        p += ((w[0] * w[1]) * w[2])[:, None] * flat[node]
    return p, torch.stack(cell, -1)


def _seed(case, seed):
    return 1000 * int(seed) + case["n"] % 997


def _pinned(*shape, dtype=F64):
    return torch.zeros(*shape, dtype=dtype, pin_memory=True)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class _Run:
    """What a program keeps between calls: the context and its page-locked output arrays."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        x = _nodes(case)
        self.ctx = PicContext(0)
        self.ctx.set_grid(x.cpu().numpy())
        self.x = x

    def field(self, u):
        self.ctx.set_ucat(u.cpu().numpy())
        self.ctx.set_dt(_dt(self.case, self.x, u))
        self.ctx.set_volume(VOLUME)

    def outputs(self, momentum):
        IM, JM, KM, n = (self.case[k] for k in ("IM", "JM", "KM", "n"))
        self.swarm = [_pinned(n, 3), _pinned(n, 3), _pinned(n, 3), _pinned(n), _pinned(n, 3, dtype=torch.int64),
                      _pinned(n, dtype=torch.int64), _pinned(n, dtype=torch.int64)]
        self.node = [_pinned(KM + 1, JM + 1, IM + 1) for _ in range(2)]
        shapes = [(KM, JM, IM + 1), (KM, JM + 1, IM), (KM + 1, JM, IM)]
        self.face = [_pinned(*s) for s in shapes]
        self.mom = [_pinned(*s, 3) for s in shapes] if momentum else []

    def check(self, rc):
        if rc:
            raise RuntimeError("%d: %s" % (rc, self.ctx.lib.fdf_GetLastError(self.ctx.h).decode()))

    def read(self):
        """The swarm, the scattered fields and the face deposits into the page-locked arrays."""
        lib, h, got = self.ctx.lib, self.ctx.h, ctypes.c_int64()
        self.check(lib.fdf_GetSwarm(h, self.case["n"], ctypes.byref(got), *[_ptr(t) for t in self.swarm]))
        self.check(lib.fdf_GetScatteredFields(h, *[_ptr(t) for t in self.node]))
        self.check(lib.fdf_GetFaceDeposits(h, *[_ptr(t) for t in self.face]))
        if self.mom:
            self.check(lib.fdf_GetFaceMomentum(h, *[_ptr(t) for t in self.mom]))
        out = dict(zip(SWARM, self.swarm), held=got.value)   # the rows past the held particles stay zero
        out.update(zip(("count", "average"), self.node))
        out.update(zip(("fi", "fj", "fk"), self.face))
        out.update(zip(("mi", "mj", "mk"), self.mom))
        return out


SWARM = ("position", "velocity", "weight", "P", "cell", "pid", "status")


def _host_swarm(case, x, seed):
    """A DMSwarm as a host code holds it between two steps: positions, cells, varying P."""
    pos, cell = _particles(case, x, case["n"], _seed(case, seed))
    P = ATMOSPHERE * (0.9 + 0.2 * _uniform01(_seed(case, seed), 9, case["n"]))
    return pos, cell, P


def _fluxes(case, x, u):
    """Contravariant face velocity, node-sized [..][3]: the face area vectors times u of the cell
    below each face (its own cell at the first face)."""
    csi, eta, zet = _metrics(x)
    own = torch.zeros_like(x)
    own[1:, 1:, 1:] = u
    own[0], own[:, 0], own[:, :, 0] = own[1], own[:, 1], own[:, :, 1]
    return torch.stack([(csi * own).sum(-1), (eta * own).sum(-1), (zet * own).sum(-1)], -1)


def _params(seed):
    """Weights as the locator's initialisation spreads them, and small biases."""
    g = torch.Generator().manual_seed(77 + int(seed))
    v = torch.rand(LOCATOR_NPARAM, generator=g, dtype=F64) * 2.0 - 1.0
    for lo, hi, s in ((0, 384, 3 ** -0.5), (384, 512, 0.1), (512, 16896, 128 ** -0.5), (16896, 17024, 0.1),
                      (17024, 33408, 128 ** -0.5), (33408, 33536, 0.1), (33536, 33920, 128 ** -0.5), (33920, 33923, 0.1)):
        v[lo:hi] *= s
    return v.to(torch.float32)


def _batch(case, seed):
    """Normalised positions and targets [batch][3] of a held-out set."""
    g = torch.Generator().manual_seed(1234 + int(seed))
    xhat = torch.rand(case["batch"], 3, generator=g, dtype=torch.float32) * 2.0 - 1.0
    t = torch.rand(case["batch"], 3, generator=g, dtype=torch.float32) * 2.0 - 1.0
    return xhat, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        n, nc = case["n"], case["ncells"]
        base = torch.arange(n, device=DEV, dtype=torch.int64) * nc // n
        far = min(case["spread"], nc - 1)
        ids = (base + torch.randint(-far, far + 1, (n,), generator=g, device=DEV)).abs()
        ids = torch.where(ids >= nc, 2 * (nc - 1) - ids, ids)
        if case["gone"]:
            ids[torch.rand(n, generator=g, device=DEV) < case["gone"]] = -1
        return dict(case=case, ids=ids.to(torch.int32), perm=torch.zeros(n, dtype=torch.int32, device=DEV),
                    start=torch.zeros(nc + 1, dtype=torch.int32, device=DEV))
    r = _Run(case, seed)
    ctx, x = r.ctx, r.x
    s = dict(case=case, run=r)
    if kind in ("simulate", "exchange", "coupled", "points"):
        u = _velocity(case, x)
        r.field(u)
        if kind != "points":
            ctx.set_form(FORMS[case["form"]])
            ctx.reserve(case["n"])
            r.outputs(case.get("momentum", False))
    if kind == "simulate":
        if case["momentum"]:
            ctx.set_momentum_deposit(True)
        if case["form"] == "learned":
            ctx.locator_train(500_000, seed=1, steps=300)
    elif kind == "exchange":
        pos, cell, P = _host_swarm(case, x, seed)
        n = case["n"]
        s["up"] = [pos.cpu().pin_memory(), torch.zeros(n, 3, dtype=F64).pin_memory(),
                   torch.zeros(n, 3, dtype=F64).pin_memory(), P.cpu().pin_memory(), cell.cpu().pin_memory(),
                   torch.arange(n).pin_memory(), torch.ones(n, dtype=torch.int64).pin_memory()]
        s["up"][1].copy_(u[tuple(cell.flip(-1).T)])
        full = torch.zeros_like(x)
        full[:-1, :-1, :-1] = u
        s["ucat"] = full.cpu().pin_memory()
    elif kind == "coupled":
        f = _fluxes(case, x, u)
        s["ucont"] = [f, 1.25 * f]
    elif kind == "points":
        pos, cell = _particles(case, x, case["n"], _seed(case, seed))
        s["pos"] = pos.cpu().numpy()
        s["hint"] = _hints(case, cell, seed).cpu().numpy() if case["hint"] else None
    elif kind in ("train", "infer"):
        s["pos"] = _particles(case, x, case["n"], _seed(case, seed))[0].cpu().numpy()
        s["seed"] = int(seed)
        if kind == "infer":
            s["params"] = _params(seed).numpy()
            s["xhat"], s["target"] = (t.numpy() for t in _batch(case, seed))
    if kind != "points":
        r.x = None
    return s


def _hints(case, cell, seed):
    """The cells the points were in before: up to two cells away per direction."""
    g = torch.Generator(device=DEV).manual_seed(50 + int(seed))
    h = cell + torch.randint(-2, 3, cell.shape, generator=g, device=DEV)
    for d, m in enumerate((case["IM"], case["JM"], case["KM"])):
        h[:, d].clamp_(0, m - 1)
    return h


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        lib = _library()
        rc = lib.fdf_SortByCell(_ptr(state["ids"]), case["n"], case["ncells"], _ptr(state["perm"]), _ptr(state["start"]),
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("fdf_SortByCell: %d" % rc)
        return {"perm": state["perm"], "start": state["start"]}
    r = state["run"]
    ctx = r.ctx
    if kind == "simulate":
        ctx.seed_particles(case["n"], _seed(case, r.seed), start_in_generating_cell=not case["corner"], P=ATMOSPHERE)
        first = ctx.initial_setup()
        log = [first.n_end]
        if case["monitor"]:
            for _ in range(case["steps"]):
                i = ctx.step()
                log += [i.n_start, i.n_end, i.removed_lost, i.removed_oob]
        else:
            ctx.steps(case["steps"])
        out = r.read()
        out["log"] = np.array(log, dtype=np.int64)
        return out
    if kind == "exchange":
        ctx.set_ucat(state["ucat"].numpy())
        r.check(ctx.lib.fdf_SetSwarm(ctx.h, case["n"], *[_ptr(t) for t in state["up"]]))
        i = ctx.step()
        out = r.read()
        out["log"] = np.array([i.n_start, i.n_end, i.removed_lost, i.removed_oob], dtype=np.int64)
        return out
    if kind == "coupled":
        ctx.seed_particles(case["n"], _seed(case, r.seed), P=ATMOSPHERE)
        ctx.initial_setup()
        for q in range(case["steps"]):
            ctx.contra2cart_device(state["ucont"][q % 2])
            ctx.step(info=False)
        out = r.read()
        out["ucat"] = ctx.get_ucat(node_sized=False)
        return out
    if kind == "points":
        cell, weight, status = ctx.locate_points(state["pos"], state["hint"])
        return {"cell": cell, "weight": weight, "status": status, "velocity": ctx.interpolate_points(cell, weight)}
    if kind == "train":
        ctx.locator_init(state["seed"])
        loss = ctx.locator_train(case["samples"], seed=state["seed"], steps=case["steps"], batch=case["batch"])
        params = ctx.locator_get_params()
        cell, y = ctx.locator_predict(state["pos"])
        return {"loss": loss, "params": params, "cell": cell, "y": y}
    ctx.locator_set_params(state["params"])
    grads, loss = ctx.locator_gradients(state["xhat"], state["target"])
    cell, y = ctx.locator_predict(state["pos"])
    return {"grads": grads, "loss": np.array([loss], dtype=np.float32), "cell": cell, "y": y}


def _library():
    from fdf_gb300 import _lib
    return _lib.load()


# ------------------------------------------------------------------ work

def work(case):
    kind, n = case["kind"], case.get("n", 0)
    nc = case.get("ncells") or case["IM"] * case["JM"] * case["KM"]
    if kind == "sort":      # ids in, permutation out, cell starts out
        return {"bytes": 8.0 * n + 4.0 * nc, "flops": 1.0 * n}
    if kind == "points":    # position, hint and outputs of both calls; the concluding cell's plane row
        return {"bytes": n * (24.0 + 24.0 + 56.0 + 48.0 + 24.0) + 24.0 * nc, "flops": 180.0 * n}
    mlp = 2.0 * (6 * 128 + 2 * 128 * 128 + 128 * 3)
    if kind == "train":     # forward and backward of every sample drawn, the weights once per step
        return {"bytes": case["steps"] * (24.0 * case["batch"] + 20.0 * 33923) + 60.0 * n,
                "flops": 3.0 * mlp * case["steps"] * case["batch"] + mlp * n}
    if kind == "infer":
        return {"bytes": 24.0 * case["batch"] + 60.0 * n + 8.0 * 33923, "flops": mlp * (3.0 * case["batch"] + n)}
    # a step reads and writes every particle's state and the grid fields once:
    # position, velocity, P, PID, cell (and the weights, written); ucat in, count, P and three faces out
    plain = case["form"] == "plain"
    state, fields = (160.0, 64.0) if plain else (116.0, 32.0)
    if case.get("momentum"):
        fields += 72.0 if plain else 36.0
    steps = 1 if kind == "exchange" else case["steps"] + 1
    out = 120.0 * n + 40.0 * nc + (72.0 * nc if case.get("momentum") else 0.0)   # the read-back
    more = {"simulate": 0.0, "exchange": 120.0 * n + 24.0 * nc, "coupled": 48.0 * nc * case.get("steps", 0)}[kind]
    return {"bytes": steps * (state * n + fields * nc) + out + more, "flops": steps * 160.0 * n}


# ------------------------------------------------------------------ what the outputs are, in 64 bits

LEFT, RIGHT, BOTTOM, TOP, FRONT, BACK = range(6)
FACES = {BACK: (0, 3, 2, 1), FRONT: (4, 7, 6, 5), BOTTOM: (0, 1, 6, 7), TOP: (3, 4, 5, 2), LEFT: (0, 7, 4, 3),
         RIGHT: (1, 2, 5, 6)}
EDGES = ((0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 7), (1, 6), (2, 5), (3, 4))
CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 1, 1), (1, 1, 1), (1, 0, 1), (0, 0, 1))


def _planes(x):
    """Per cell (i fastest): six faces' centroid and unit normal away from the cell's centre or along its edges'
    order, and the distance below which a point is on a face."""
    KM, JM, IM = (s - 1 for s in x.shape[:3])
    rows = torch.empty(KM, JM, IM, 37, dtype=F64, device=DEV)
    for k0 in range(0, KM, 64):
        k1 = min(KM, k0 + 64)
        v = [x[k0 + c[2]:k1 + c[2], c[1]:JM + c[1], c[0]:IM + c[0]] for c in CORNERS]
        total = 0.0
        for a, b in EDGES:
            d = v[b] - v[a]
            total = total + torch.sqrt(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2])
        rows[k0:k1, ..., 36] = 1e-11 * (total / 12.0)
        centre = v[0]
        for q in range(1, 8):
            centre = centre + v[q]
        centre = centre / 8.0
        for f, (p, q, r, s) in FACES.items():
            e1, e2 = v[q] - v[p], v[s] - v[p]
            n = torch.stack([e1[..., 1] * e2[..., 2] - e1[..., 2] * e2[..., 1],
                             e1[..., 2] * e2[..., 0] - e1[..., 0] * e2[..., 2],
                             e1[..., 0] * e2[..., 1] - e1[..., 1] * e2[..., 0]], -1)
            mag = torch.sqrt(n[..., 0] * n[..., 0] + n[..., 1] * n[..., 1] + n[..., 2] * n[..., 2])
            fc = 0.25 * (((v[p] + v[q]) + v[r]) + v[s])
            t = centre - fc
            dot = n[..., 0] * t[..., 0] + n[..., 1] * t[..., 1] + n[..., 2] * t[..., 2]
            n = torch.where((dot > 1e-9)[..., None], -n, n) / mag[..., None]
            rows[k0:k1, ..., 6 * f:6 * f + 3] = fc
            rows[k0:k1, ..., 6 * f + 3:6 * f + 6] = n
    return rows.reshape(-1, 37)


def _walk(dims, rows, pos, cell):
    """The walking search from each point's cell: (cell or -1, weights), both for the points given."""
    IM, JM, KM = dims
    ijk = torch.stack([cell % IM, (cell // IM) % JM, cell // (IM * JM)], -1)
    ijk[cell < 0] = 0
    found = torch.full_like(cell, -1)
    dist = torch.zeros(len(pos), 6, dtype=F64, device=DEV)
    live, saved = torch.arange(len(pos), device=DEV), torch.full_like(cell, -1)
    power = lam = 1
    for step in range(1000):
        q = ijk[live]
        inside = ((q >= 0) & (q < torch.tensor([IM, JM, KM], device=DEV))).all(-1)
        live, q = live[inside], q[inside]
        cur = (q[:, 2] * JM + q[:, 1]) * IM + q[:, 0]
        if step > 16:   # a cell met again: the walk goes round until it is given up
            again = cur == saved[live]
            live, q, cur = live[~again], q[~again], cur[~again]
            if step >= power:
                saved[live] = cur
                power *= 2
        else:
            power = 32
        if not len(live):
            break
        row, p = rows[cur], pos[live]
        d = torch.stack([((row[:, 6 * f] - p[:, 0]) * row[:, 6 * f + 3] + (row[:, 6 * f + 1] - p[:, 1]) * row[:, 6 * f + 4])
                         + (row[:, 6 * f + 2] - p[:, 2]) * row[:, 6 * f + 5] for f in range(6)], -1)
        d = torch.where(d.abs() < row[:, 36:], torch.zeros_like(d), d)
        neg = d < 0
        done = ~neg.any(-1) | (d == 0).any(-1)
        found[live[done]] = cur[done]
        dist[live[done]] = d[done]
        live, q, neg = live[~done], q[~done], neg[~done].to(torch.int64)
        pick = lambda a, b: neg[:, a] - (1 - neg[:, a]) * neg[:, b]  # noqa: E731
        ijk[live] = q + torch.stack([-pick(LEFT, RIGHT), -pick(BOTTOM, TOP), pick(FRONT, BACK)], -1)
    d = torch.where(dist <= 1e-14, torch.full_like(dist, 1e-14), dist)
    w = torch.stack([d[:, LEFT] / (d[:, LEFT] + d[:, RIGHT]), d[:, BOTTOM] / (d[:, BOTTOM] + d[:, TOP]),
                     d[:, BACK] / (d[:, FRONT] + d[:, BACK])], -1)
    return found, w


def _corners(u):
    """The node field: the mean of a node's adjacent cells."""
    KM, JM, IM = u.shape[:3]
    acc = torch.zeros(KM + 1, JM + 1, IM + 1, 3, dtype=F64, device=DEV)
    num = torch.zeros(KM + 1, JM + 1, IM + 1, 1, dtype=F64, device=DEV)
    for dk in (1, 0):
        for dj in (1, 0):
            for di in (1, 0):
                at = (slice(dk, KM + dk), slice(dj, JM + dj), slice(di, IM + di))
                acc[at] += u
                num[at] += 1.0
    return acc / num


def _interpolate(dims, corner, cell, w):
    IM, JM, KM = dims
    flat, mx, my = corner.reshape(-1, 3), IM + 1, JM + 1
    c = cell.clamp(min=0)
    q0 = ((c // (IM * JM)) * my + (c // IM) % JM) * mx + c % IM
    a = w.clamp(0.0, 1.0)
    o = 1.0 - a
    v, sw = torch.zeros(len(cell), 3, dtype=F64, device=DEV), torch.zeros(len(cell), dtype=F64, device=DEV)
    for k in range(8):
        b = (k & 1, (k >> 1) & 1, (k >> 2) & 1)
        t = [a[:, d] if b[d] else o[:, d] for d in range(3)]
        t = (t[0] * t[1]) * t[2]
        v += t[:, None] * flat[q0 + (b[2] * my + b[1]) * mx + b[0]]
        sw += t
    v /= sw[:, None]
    return torch.where((cell >= 0)[:, None], v, torch.zeros_like(v))


def _deposit(dims, cell, w, P, vel, momentum):
    """ParticleCount, mean P, the three face volumes and, where asked, the face momenta."""
    IM, JM, KM = dims
    ok = cell >= 0
    cell, w, P, vel = cell[ok], w[ok], P[ok], vel[ok]
    nc = IM * JM * KM
    num = torch.bincount(cell, minlength=nc).to(F64)
    psum = torch.zeros(nc, dtype=F64, device=DEV).index_add_(0, cell, P)
    node = []
    for v in (num, torch.where(num > 0, psum / num.clamp(min=1.0), psum)):
        full = torch.zeros(KM + 1, JM + 1, IM + 1, dtype=F64, device=DEV)
        full[:KM, :JM, :IM] = v.reshape(KM, JM, IM)
        node.append(full)
    i, j, k = cell % IM, (cell // IM) % JM, cell // (IM * JM)
    lower = [(k * JM + j) * (IM + 1) + i, (k * (JM + 1) + j) * IM + i, cell]
    stride, third = (1, IM, IM * JM), VOLUME / 3.0
    shapes = [(KM, JM, IM + 1), (KM, JM + 1, IM), (KM + 1, JM, IM)]
    face, mom = [], []
    for d in range(3):
        size = math.prod(shapes[d])
        hi, lo = w[:, d] * third, (1.0 - w[:, d]) * third
        face.append(torch.zeros(size, dtype=F64, device=DEV).index_add_(0, lower[d] + stride[d], hi)
                    .index_add_(0, lower[d], lo).reshape(shapes[d]))
        if momentum:
            mom.append(torch.zeros(size, 3, dtype=F64, device=DEV).index_add_(0, lower[d] + stride[d], hi[:, None] * vel)
                       .index_add_(0, lower[d], lo[:, None] * vel).reshape(*shapes[d], 3))
    return node + face + mom


def _metrics(x):
    """Face area vectors Csi, Eta, Zet, node-sized, extended to the first faces of the other directions."""
    csi, eta, zet = (torch.zeros_like(x) for _ in range(3))
    dj = 0.5 * (x[1:, 1:] + x[:-1, 1:] - x[1:, :-1] - x[:-1, :-1])
    dk = 0.5 * (x[1:, :-1] + x[1:, 1:] - x[:-1, :-1] - x[:-1, 1:])
    csi[1:, 1:] = torch.linalg.cross(dj, dk)
    di = 0.5 * (x[1:, :, 1:] + x[:-1, :, 1:] - x[1:, :, :-1] - x[:-1, :, :-1])
    dk = 0.5 * (x[1:, :, 1:] + x[1:, :, :-1] - x[:-1, :, 1:] - x[:-1, :, :-1])
    eta[1:, :, 1:] = torch.linalg.cross(dk, di)
    di = 0.5 * (x[:, 1:, 1:] + x[:, :-1, 1:] - x[:, 1:, :-1] - x[:, :-1, :-1])
    dj = 0.5 * (x[:, 1:, 1:] + x[:, 1:, :-1] - x[:, :-1, 1:] - x[:, :-1, :-1])
    zet[:, 1:, 1:] = torch.linalg.cross(di, dj)
    # node 0 takes node 1, then the last node the one before it, direction by direction
    for d, fields in ((2, (eta, zet)), (1, (csi, zet)), (0, (csi, eta))):
        for v in fields:
            v.select(d, 0).copy_(v.select(d, 1))
            v.select(d, -1).copy_(v.select(d, -2))
    return csi, eta, zet


def _cartesian(csi, eta, zet, f, u):
    """u with its interior cells set from the face velocity f, by Cramer's rule on the face-averaged metrics."""
    m = torch.stack([0.5 * (csi[1:-1, 1:-1, :-2] + csi[1:-1, 1:-1, 1:-1]),
                     0.5 * (eta[1:-1, :-2, 1:-1] + eta[1:-1, 1:-1, 1:-1]),
                     0.5 * (zet[:-2, 1:-1, 1:-1] + zet[1:-1, 1:-1, 1:-1])], -2)
    q = torch.stack([0.5 * (f[1:-1, 1:-1, :-2, 0] + f[1:-1, 1:-1, 1:-1, 0]),
                     0.5 * (f[1:-1, :-2, 1:-1, 1] + f[1:-1, 1:-1, 1:-1, 1]),
                     0.5 * (f[:-2, 1:-1, 1:-1, 2] + f[1:-1, 1:-1, 1:-1, 2])], -1)
    a, b, c = m[..., 0, :], m[..., 1, :], m[..., 2, :]
    bc, ca, ab = torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)
    det = (a * bc).sum(-1, keepdim=True)
    out = u.clone()
    out[1:, 1:, 1:] = (q[..., 0:1] * bc + q[..., 1:2] * ca + q[..., 2:3] * ab) / det
    return out


def _chunks(n, size=1 << 21):
    return [slice(a, min(n, a + size)) for a in range(0, n, size)]


class _Swarm:
    """The path's stages in 64 bits on a swarm held in the plain form's order."""

    def __init__(self, case, x, pos, cell, P, vel=None):
        self.dims = (case["IM"], case["JM"], case["KM"])
        self.case, self.rows = case, _planes(x)
        self.lo, self.hi = x.reshape(-1, 3).amin(0) - 1e-6, x.reshape(-1, 3).amax(0) + 1e-6
        self.pos, self.cell, self.P = pos, cell, P
        self.vel = torch.zeros_like(pos) if vel is None else vel
        self.w = torch.zeros_like(pos)
        self.pid = torch.arange(len(pos), device=DEV)

    def locate(self, drop):
        cell, w = torch.empty_like(self.cell), torch.empty_like(self.w)
        for s in _chunks(len(self.pos)):
            cell[s], w[s] = _walk(self.dims, self.rows, self.pos[s], self.cell[s])
        self.w = torch.where((cell >= 0)[:, None], w, self.w)
        self.cell = cell
        keep = torch.ones_like(cell, dtype=torch.bool)
        if drop:
            keep = (cell >= 0) & (self.pos >= self.lo).all(-1) & (self.pos <= self.hi).all(-1)
        last = math.prod(self.dims)
        key = torch.where(self.cell < 0, torch.full_like(self.cell, last), self.cell)
        order = torch.argsort(self.pid)
        order = order[torch.argsort(key[order], stable=True)]
        order = order[keep[order]]
        for f in ("pos", "cell", "P", "vel", "w", "pid"):
            setattr(self, f, getattr(self, f)[order])

    def interpolate(self, u):
        corner = _corners(u)
        self.vel = torch.cat([_interpolate(self.dims, corner, self.cell[s], self.w[s]) for s in _chunks(len(self.cell))]
                             or [self.vel])

    def step(self, u, dt):
        self.pos = self.pos + self.vel * dt
        self.locate(True)
        self.interpolate(u)

    def answer(self, momentum, held):
        out = dict.fromkeys(SWARM)
        if held:   # the order of the held particles is the plain form's
            for k, v in (("position", self.pos), ("velocity", self.vel), ("weight", self.w), ("P", self.P)):
                out[k] = torch.zeros(self.case["n"], *v.shape[1:], dtype=F64, device=DEV)
                out[k][:len(v)] = v
        names = ("count", "average", "fi", "fj", "fk") + (("mi", "mj", "mk") if momentum else ())
        out.update(zip(names, _deposit(self.dims, self.cell, self.w, self.P, self.vel, momentum)))
        return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sort", "train"):   # whole numbers; a training's path is not a value
        return None
    x = _nodes(case)
    dims = (case["IM"], case["JM"], case["KM"])
    if kind == "infer":
        return _exact_infer(case, seed, x)
    u = _velocity(case, x)
    dt = _dt(case, x, u)
    if kind == "points":
        pos, cell = _particles(case, x, case["n"], _seed(case, seed))
        start = torch.zeros(case["n"], dtype=torch.int64, device=DEV)
        if case["hint"]:
            h = _hints(case, cell, seed)
            start = (h[:, 2] * dims[1] + h[:, 1]) * dims[0] + h[:, 0]
        found, w = _walk(dims, _planes(x), pos, start)
        w = torch.where((found >= 0)[:, None], w, torch.zeros_like(w))
        return {"cell": None, "weight": w, "status": None, "velocity": _interpolate(dims, _corners(u), found, w)}
    if kind == "exchange":
        pos, cell, P = _host_swarm(case, x, seed)
        vel = u[tuple(cell.flip(-1).T)].clone()
        s = _Swarm(case, x, pos, (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0], P, vel)
        s.step(u, dt)
        return s.answer(False, case["form"] == "plain")
    if case["n"] * case["steps"] > 4e8:   # over 20 seconds in this way
        return None
    pos, cell = _particles(case, x, case["n"], _seed(case, seed))
    cell = (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
    if case.get("corner"):
        cell = torch.full_like(cell, -1)
    s = _Swarm(case, x, pos, cell, torch.full_like(pos[:, 0], ATMOSPHERE))
    s.locate(False)
    s.interpolate(u)
    if kind == "coupled":
        m, f = _metrics(x), _fluxes(case, x, u)
    for q in range(case["steps"]):
        if kind == "coupled":
            u = _cartesian(*m, f if q % 2 == 0 else 1.25 * f, u)
        s.step(u, dt)
    out = s.answer(case.get("momentum", False), case["form"] == "plain")
    if kind == "coupled":
        out["ucat"] = u
    return out


def _exact_infer(case, seed, x):
    p = _params(seed).to(DEV, F64).requires_grad_(True)
    sizes = ((0, 384, 512, 3), (512, 16896, 17024, 128), (17024, 33408, 33536, 128), (33536, 33920, 33923, 128))

    def net(h):
        for L, (a, b, c, k) in enumerate(sizes):
            h = h @ p[a:b].reshape(-1, k).T + p[b:c]
            if L < 3:
                h = h * torch.sigmoid(h)
        return h

    xhat, t = (v.to(DEV, F64) for v in _batch(case, seed))
    scale = torch.tensor([case["IM"], case["JM"], case["KM"]], dtype=F64, device=DEV) / 2.0
    loss = (((net(xhat) - t) * scale) ** 2).sum(-1).div(3.0).mean()
    (grad,) = torch.autograd.grad(loss, p)
    lo, hi = x.reshape(-1, 3).amin(0) - 1e-6, x.reshape(-1, 3).amax(0) + 1e-6
    pos = _particles(case, x, case["n"], _seed(case, seed))[0]
    with torch.no_grad():
        y = torch.cat([net((pos[s] - 0.5 * (lo + hi)) * (2.0 / (hi - lo))) for s in _chunks(case["n"])])
    return {"grads": grad.detach(), "loss": loss.detach().reshape(1), "cell": None, "y": y}
