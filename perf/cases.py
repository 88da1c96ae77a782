"""The performance cases: what a user's program has this library do, through
its public entry points (vof_b200.Solver and vof_b200.slab), from one step of
a small box to the largest runs.

A pass of a forward case is a restart: the five state fields are set from the
caller's arrays, `steps` time steps are run, and the five fields are read
back.  An adjoint case records the steps, reverses them and reads the
gradients of all five fields back.  The sizes are those of the benchmark
(200^3, the 64^3 adjoint), of the tests (24x20x16, 32^3) and generic ones, odd
and ragged sizes among them.

exact() restates the step (and, for the adjoint, its derivative by automatic
differentiation) in plain torch operations in 64 bits.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "cuda-lbm-ibm-fvm_b200"))

import vof_b200 as V  # noqa: E402
from vof_b200 import slab  # noqa: E402

STATE = ("F", "u", "v", "w", "p")
MODES = {"plain": V.MODE_PLAIN, "mixed": V.MODE_MIXED, "fp64": V.MODE_FP64}


def _case(name, kind, nx, ny, nz, steps, iters=10, mode="plain", start="rest", csf=False, host=False, volume="none",
          ranks=1):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "iters": iters, "mode": mode, "start": start,
         "csf": csf, "host": host, "volume": volume, "ranks": ranks}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small box stepped one call at a time by a program that looks at the liquid volume after every step
        # (the size of the smoke test): launch latency and the wait for the value
        _case("monitor_24x20x16", "run", 24, 20, 16, 6, start="flow", volume="blocking"),
        # the 32^3 dam break of the golden data, a batch of steps between two looks at the fields
        _case("run_32", "run", 32, 32, 32, 30),
        # 64^3 from numpy arrays and back, the way a Python program without torch uses the library
        _case("run_64_host", "run", 64, 64, 64, 30, start="flow", host=True),
        # the benchmark: the 200^3 dam break from rest, the volume of every step written to pinned memory
        _case("run_200", "run", 200, 200, 200, 12, volume="async"),
        # a ragged box in full flow
        _case("run_201x157x93", "run", 201, 157, 93, 12, start="flow"),
        # the largest plain run: every field is twice the size of the L2
        _case("run_400", "run", 400, 400, 400, 4, start="flow"),
        # the surface-tension option
        _case("csf_128", "run", 128, 128, 128, 8, start="flow", csf=True),
        # convergent pressure, mixed-precision solver, the benchmark's size
        _case("mixed_200", "run", 200, 200, 200, 2, mode="mixed"),
        # convergent pressure in FP64 on a box of unequal sides
        _case("fp64_100x80x126", "run", 100, 80, 126, 2, mode="fp64", start="flow"),
        # gradient of the liquid volume in a box with respect to the initial state: the benchmark's 64^3
        _case("adjoint_64", "adjoint", 64, 64, 64, 40, start="flow"),
        # the same on a grid large enough to fill the GPU
        _case("adjoint_144x136x150", "adjoint", 144, 136, 150, 24, start="flow"),
        # z slabs with their halo exchange after every step, two ranks in one process
        _case("slab_160x120x200", "slab", 160, 120, 200, 8, ranks=2, volume="blocking"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, lo, hi):
    """A side that the multigrid hierarchy coarsens: at most 8 times a power of two, 3, 5 or 7 times one."""
    while True:
        n = rng.choice((1, 3, 5, 7, 9, 15, 25)) << rng.randrange(0, 8)
        if lo <= n <= hi:
            return n


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "csf", "host", "mixed", "fp64", "adjoint", "slab"))
    start = rng.choice(("rest", "flow"))
    cells = math.exp(rng.uniform(math.log(4e3), math.log(5e7)))  # about so many cells in all
    if kind in ("mixed", "fp64"):
        base = math.exp(rng.uniform(math.log(30), math.log(155)))  # cells near to cubes, as the solver wants them
        n = [_smooth(rng, base / 1.3, base * 1.3) for _ in range(3)]
        return _case("", "run", *n, rng.randint(1, 2), mode=kind, start=start)
    if kind == "adjoint":
        n = [_log_int(rng, 20, 140) for _ in range(3)]
        return _case("", "adjoint", *n, rng.randint(4, 24), iters=rng.choice((4, 10, 10)), start="flow")
    if kind == "slab":
        return _case("", "slab", _log_int(rng, 40, 200), _log_int(rng, 40, 200), _log_int(rng, 80, 220),
                     rng.randint(3, 8), ranks=2, volume="blocking", start=start)
    side = cells ** (1.0 / 3.0)
    a, b = math.exp(rng.uniform(-0.4, 0.4)), math.exp(rng.uniform(-0.4, 0.4))
    n = [max(8, min(420, int(round(side * f)))) for f in (a, b, 1.0 / (a * b))]
    if kind == "host":
        n = [min(x, 130) for x in n]
    total = n[0] * n[1] * n[2]
    if kind == "csf" and total > 2e7:
        n = [max(8, x // 2) for x in n]
        total = n[0] * n[1] * n[2]
    steps = max(1, min(30, int(2e8 / total / 2)))
    steps = rng.randint(max(1, steps // 2), steps)
    # (an odd number of sweeps feeds the alternating pressure mode from step to step: for few steps only)
    iters = rng.choice((4, 10, 10, 10, 20) if steps > 4 else (3, 7, 10, 10, 10, 15))
    return _case("", "run", *n, steps, iters=iters, start=start, csf=kind == "csf",
                 host=kind == "host", volume=rng.choice(("none", "async", "blocking")))


# ---- inputs ------------------------------------------------------------------
def _params(c):
    return V.default_params(c["nx"], c["ny"], c["nz"], gy=0.0, gz=-9.81, jacobi_iters=c["iters"],
                            mode=MODES[c["mode"]], surface_tension=int(c["csf"]))


def _fields(c, seed):
    """The initial state on the GPU, float32, (nz+2, ny+2, nx+2): a block of liquid (a dam) with a rough surface, at
    rest, or in flow: smooth velocities of some tenths of a metre a second, hydrostatic pressure and a wave of it."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    dev = {"device": "cuda", "dtype": torch.float32}
    # cell centres in units of the box, ghosts included
    x = ((torch.arange(nx + 2, **dev) - 0.5) / nx).view(1, 1, -1)
    y = ((torch.arange(ny + 2, **dev) - 0.5) / ny).view(1, -1, 1)
    z = ((torch.arange(nz + 2, **dev) - 0.5) / nz).view(-1, 1, 1)
    xw, yw = 0.4 + 0.1 * rng.uniform(-1, 1), 0.4 + 0.1 * rng.uniform(-1, 1)
    if c["start"] == "rest":
        h = 0.6 + (0.5 / nz) * (2 * torch.rand((1, ny + 2, nx + 2), generator=gen, **dev) - 1)
    else:
        h = 0.6 + 0.05 * torch.sin(2 * math.pi * x + rng.uniform(0, 6)) * torch.cos(2 * math.pi * y + rng.uniform(0, 6))
    F = torch.clamp((h - z) * nz + 0.5, 0.0, 1.0)
    F = F * torch.clamp((xw - x) * nx + 0.5, 0.0, 1.0) * torch.clamp((yw - y) * ny + 0.5, 0.0, 1.0)
    s = {"F": bc_F(F.contiguous())}
    zero = torch.zeros_like(F)
    if c["start"] == "rest":
        return {**s, "u": zero, "v": zero.clone(), "w": zero.clone(), "p": zero.clone()}
    xf, yf, zf = x - 0.5 / nx, y - 0.5 / ny, z - 0.5 / nz  # the faces below the cells

    def vel(along, c1, c2):
        a, b, ph, ps, k = (rng.uniform(0.1, 0.3), rng.uniform(0.02, 0.1), rng.uniform(0, 6, 2), rng.uniform(0, 6, 2),
                           rng.integers(1, 4, 3))
        return (a * torch.sin(math.pi * along) * torch.cos(math.pi * c1 + ph[0]) * torch.cos(math.pi * c2 + ph[1]) +
                b * torch.sin(2 * math.pi * int(k[0]) * along) * torch.sin(2 * math.pi * int(k[1]) * c1 + ps[0]) *
                torch.sin(2 * math.pi * int(k[2]) * c2 + ps[1])).contiguous()

    u, v, w = vel(xf, y, z), vel(yf, x, z), vel(zf, x, y)
    u, v, w = bc_velocity(u, v, w)
    ph = rng.uniform(0, 6, 3)
    p = 588.6 * torch.clamp(0.6 - z, min=0.0) / 0.6 + rng.uniform(10, 30) * torch.cos(math.pi * x + ph[0]) * torch.cos(
        math.pi * y + ph[1]) * torch.cos(math.pi * z + ph[2])
    q = torch.zeros_like(F)
    q[1:-1, 1:-1, 1:-1] = p[1:-1, 1:-1, 1:-1]
    return {**s, "u": u.contiguous(), "v": v.contiguous(), "w": w.contiguous(), "p": q}


def _box(c):
    return (0.031, 0.083, 0.012, 0.077, 0.0, 0.0413)


def prepare(case, seed):
    c = dict(case)
    prm = _params(c)
    f = _fields(c, seed)
    st = {"case": c}
    if c["host"]:
        st["in"] = {k: x.cpu().numpy() for k, x in f.items()}
    else:
        st["in"] = f
    if c["kind"] == "slab":
        st["group"] = slab.LocalGroup(prm, c["ranks"], lambda q: V.Solver(q), device="cuda")
        parts = [r.slab for r in st["group"].ranks]
        st["in"] = [{k: x[s.lo - 1:s.hi + 2].contiguous() for k, x in f.items()} for s in parts]
        st["out"] = {k: torch.empty_like(x) for k, x in f.items()}
        return st
    st["solver"] = V.Solver(prm)
    if c["kind"] == "run" and not c["host"]:
        st["out"] = {k: torch.empty_like(x) for k, x in f.items()}
    if c["volume"] == "async":
        st["volumes"] = torch.zeros(c["steps"], dtype=torch.float64).pin_memory()
    return st


# ---- one pass ------------------------------------------------------------------
def _run_forward(st):
    c, s = st["case"], st["solver"]
    if c["host"]:
        s.upload_state(**st["in"])
    else:
        for k, x in st["in"].items():
            s.upload(k, device_ptr=x.data_ptr())
    volumes = None
    if c["volume"] == "none":
        s.run(1, c["steps"])
    elif c["volume"] == "async":
        volumes = st["volumes"]
        for n in range(c["steps"]):
            s.run(1 + n, 1)
            s.reduce_async("volume", volumes.data_ptr() + 8 * n)
    else:
        volumes = []
        for n in range(c["steps"]):
            s.step(1 + n)
            volumes.append(s.reduce("volume"))
    if c["host"]:
        out = s.state()
    else:
        out = st["out"]
        for k, x in out.items():
            s.download_device(k, x.data_ptr())
    return {"state": out, "volumes": volumes}


def _run_adjoint(st):
    c, s = st["case"], st["solver"]
    for k, x in st["in"].items():
        s.upload(k, device_ptr=x.data_ptr())
    s.forward_record(1, c["steps"])
    r = s.backward(_box(c))
    return {"loss": r["loss"], "grad_g": r["grad_g"], "grad": {k: s.adjoint(k) for k in STATE}}


def _run_slab(st):
    c, g = st["case"], st["group"]
    for r, part in zip(g.ranks, st["in"]):
        for k, x in part.items():
            r.engine.upload(k, device_ptr=x.data_ptr())
    g.run(1, c["steps"])
    volume = g.volume()
    for r in g.ranks:  # the planes that each rank owns, with the ghost planes at the two ends of the box
        a, b = r.slab.own0 - (r.comm.rank == 0), r.slab.own1 + (r.comm.rank == c["ranks"] - 1)
        for k, x in st["out"].items():
            r.engine.get_planes(k, r.slab.local(a), b - a + 1, device_ptr=x[a].data_ptr())
    return {"state": st["out"], "volume": volume}


def run(state):
    return {"run": _run_forward, "adjoint": _run_adjoint, "slab": _run_slab}[state["case"]["kind"]](state)


def work(case):
    """A step reads its five state fields and writes them (40 bytes a cell), the convergent modes' FP64 pressure besides;
    a reversed step does so for the five FP64 adjoint fields and reads the state it reverses (100 bytes a cell).
    Operations: those of the step's expressions, the FCT stages and `iters` pressure sweeps (the convergent modes: what
    one multigrid cycle per digit pair of its tolerance takes at least)."""
    c = case
    cells = float(c["nx"]) * c["ny"] * c["nz"]
    per_step, flops = 40.0, 130.0 + 12.0 + 14.0 * c["iters"] + 30.0 + 3 * 60.0
    if c["mode"] != "plain":
        per_step += 16.0
        flops += 4 * 100.0 - 14.0 * c["iters"]
    if c["csf"]:
        flops += 80.0
    if c["kind"] == "adjoint":
        per_step += 100.0
        flops *= 3.0
    return {"bytes": cells * (c["steps"] * per_step + (60.0 if c["kind"] == "adjoint" else 40.0)),
            "flops": cells * c["steps"] * flops}


# ---- the step restated in torch ----------------------------------------------------
# Arrays are (nz+2, ny+2, nx+2).  Every non-smooth choice goes through a _Switch, which can hand the choices of an
# FP32 evaluation to an FP64 one, and so do the values that derivatives are taken at (the adjoint differentiates the
# side that the FP32 forward took, at the FP32 forward's values).
class _Put(torch.autograd.Function):
    """The value of `y`, with the derivative of `x`."""

    @staticmethod
    def forward(ctx, x, y):
        return y.to(x.dtype)

    @staticmethod
    def backward(ctx, grad):
        return grad, None


class _Switch:
    def __init__(self, tape=None):
        self.tape, self.out, self.at = tape, [], 0

    def __call__(self, cond):
        if self.tape is None:
            self.out.append(cond)
            return cond
        cond = self.tape[self.at]
        self.at += 1
        return cond

    def value(self, x):
        if self.tape is None:
            self.out.append(x)
            return x
        self.at += 1
        return _Put.apply(x, self.tape[self.at - 1])

    def pick(self, cond, a, b):
        return torch.where(self(cond), a, b)

    def mx(self, a, b):
        return self.pick(a >= b, a, b)

    def mn(self, a, b):
        return self.pick(a <= b, a, b)


class _Plain(_Switch):
    """Choices as they fall, none kept."""

    def __call__(self, cond):
        return cond

    def value(self, x):
        return x


def bc_F(F):
    F[:, 0, :] = F[:, 1, :]
    F[:, -1, :] = F[:, -2, :]
    F[:, :, 0] = F[:, :, 1]
    F[:, :, -1] = F[:, :, -2]
    F[0] = F[1]
    F[-1] = F[-2]
    return F


def bc_velocity(u, v, w):
    """Free slip, as three passes along j, i and k."""
    u, v, w = u.clone(), v.clone(), w.clone()
    for a in (u, w):
        a[:, 0, :] = a[:, 1, :]
        a[:, -1, :] = a[:, -2, :]
    v[:, 1, :] = 0
    v[:, -1, :] = 0
    for a in (v, w):
        a[:, :, 0] = a[:, :, 1]
        a[:, :, -1] = a[:, :, -2]
    u[:, :, 1] = 0
    u[:, :, -1] = 0
    for a in (u, v):
        a[0] = a[1]
        a[-1] = a[-2]
    w[1] = 0
    w[-1] = 0
    return u, v, w


class _Step:
    """One time step in the precision of `dtype`."""

    def __init__(self, c, dtype, device):
        f = np.float32
        n = (c["nx"], c["ny"], c["nz"])
        d = [f(f(0.1) / f(x)) for x in n]
        di = [f(f(1.0) / x) for x in d]

        def t(v):  # a tensor: torch divides by a Python number by multiplying with its reciprocal
            return torch.tensor(float(v), dtype=dtype, device=device)

        self.c, self.n, self.dtype, self.device = c, n, dtype, device
        self.d, self.di = [t(x) for x in d], [t(x) for x in di]
        self.dt = t(f(4.0e-6))
        self.rho_l, self.rho_g, self.nu_l, self.nu_g = t(1000.0), t(50.0), t(f(1.0e-6)), t(f(1.5e-5))
        self.sigma = t(f(0.007))
        self.g = [t(0.0), t(0.0), t(f(-9.81))]
        self.one, self.zero = t(1.0), t(0.0)

    def at(self, a, x=0, y=0, z=0):
        nx, ny, nz = self.n
        return a[1 + z:1 + z + nz, 1 + y:1 + y + ny, 1 + x:1 + x + nx]

    def clamp01(self, sw, v):
        return self.zero + self.one + v - sw.mx(self.one, v) - sw.mn(self.zero, v)

    def rho_nu(self, sw, F):
        f = self.clamp01(sw, F)
        return self.rho_g * (1.0 - f) + self.rho_l * f, self.nu_l * f + self.nu_g * (1.0 - f)

    def _shift(self, axis, by):
        return {"xyz"[axis]: by}

    def star(self, sw, vel, axis, nu):
        """The predicted velocity along `axis`, interior cells."""
        a = vel[axis]
        at = self.at
        ac = at(a)
        conv = []
        for q in range(3):  # the velocity along q at this face
            if q == axis:
                conv.append(ac)
                continue
            b, m, up = vel[q], self._shift(axis, -1), self._shift(q, 1)
            # (the reference's order of the four terms)
            if axis == 0:
                four = (at(b, **m), at(b, **m, **up), at(b), at(b, **up))
            elif axis == 1 and q == 0:
                four = (at(b, **m), at(b), at(b, **m, **up), at(b, **up))
            elif axis == 1:
                four = (at(b, **m, **up), at(b, **m), at(b), at(b, **up))
            elif q == 0:
                four = (at(b, **m, **up), at(b, **m), at(b, **up), at(b))
            else:
                four = (at(b, **m, **up), at(b, **m), at(b), at(b, **up))
            conv.append(0.25 * (four[0] + four[1] + four[2] + four[3]))
        visc = adv = None
        for q in range(3):
            lo, hi = at(a, **self._shift(q, -1)), at(a, **self._shift(q, 1))
            grad = sw.pick(conv[q] > 0, (ac - lo) * self.di[q], (hi - ac) * self.di[q])
            vq = nu * (lo - 2.0 * ac + hi) * self.di[q] * self.di[q]
            visc = vq if visc is None else visc + vq
            adv = -conv[q] * grad if adv is None else adv - conv[q] * grad
        return ac + self.dt * (visc + adv + self.g[axis])

    def only(self, a, axis):
        """Zero on the first face along `axis`, in an array with zero ghosts."""
        full = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
        keep = torch.ones_like(full)
        keep.select(2 - axis, 1).fill_(0)
        return full * keep

    def csf(self, F):
        nx, ny, nz = self.n
        h = [0.5 * x for x in self.di]
        gr = [(self.at(F, **self._shift(q, 1)) - self.at(F, **self._shift(q, -1))) * h[q] for q in range(3)]
        mag = torch.sqrt(gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2])
        has = mag > 1e-6 * self.di[0]
        safe = torch.where(has, mag, self.one)
        normal = [torch.where(has, x / safe, self.zero) for x in gr]
        parts = []
        for q in range(3):
            dim = 2 - q
            a = normal[q]
            first, last = a.narrow(dim, 0, 1), a.narrow(dim, self.n[q] - 1, 1)
            e = torch.cat((a.narrow(dim, 1, self.n[q] - 1), -last), dim)
            w = torch.cat((-first, a.narrow(dim, 0, self.n[q] - 1)), dim)
            parts.append((e - w) * h[q])
        return torch.nn.functional.pad(-(parts[0] + parts[1] + parts[2]), (1, 1, 1, 1, 1, 1))

    def pressure(self, p, rhs):
        """`iters` Jacobi sweeps with zero-gradient walls."""
        cc = [x * x for x in self.di]
        walls = []
        for q in range(3):
            shape = [1, 1, 1]
            shape[2 - q] = self.n[q]
            hi = cc[q].expand(shape).clone()
            lo = cc[q].expand(shape).clone()
            hi.select(2 - q, self.n[q] - 1).fill_(0)
            lo.select(2 - q, 0).fill_(0)
            walls.append((lo, hi))
        (aw, ae), (as_, an), (ab, af) = walls
        ap = -(ae + aw + an + as_ + af + ab)
        at = self.at
        for _ in range(self.c["iters"]):
            p = torch.nn.functional.pad((rhs - ae * at(p, x=1) - aw * at(p, x=-1) - an * at(p, y=1) -
                                         as_ * at(p, y=-1) - af * at(p, z=1) - ab * at(p, z=-1)) / ap,
                                        (1, 1, 1, 1, 1, 1))
        return p

    def solved(self, rhs):
        """The exact solution of the mean-free Neumann system, of mean zero: cosine transforms along each axis."""
        b = (rhs - rhs.mean()).double()
        lam = 0.0
        basis = []
        for q in range(3):
            n = self.n[q]
            i = torch.arange(n, dtype=torch.float64, device=self.device)
            m = torch.cos(math.pi * i.view(-1, 1) * (i.view(1, -1) + 0.5) / n) * math.sqrt(2.0 / n)
            m[0] *= math.sqrt(0.5)
            shape = [1, 1, 1]
            shape[2 - q] = n
            dq = float(self.di[q])
            lam = lam + (2 * dq * dq * (torch.cos(math.pi * i / n) - 1.0)).view(shape)
            basis.append(m)
        t = torch.einsum("ai,kji->kja", basis[0], b)
        t = torch.einsum("bj,kja->kba", basis[1], t)
        t = torch.einsum("ck,kba->cba", basis[2], t)
        lam[0, 0, 0] = 1.0
        t = t / lam
        t[0, 0, 0] = 0.0
        t = torch.einsum("ck,cba->kba", basis[2], t)
        t = torch.einsum("bj,kba->kja", basis[1], t)
        t = torch.einsum("ai,kja->kji", basis[0], t)
        return torch.nn.functional.pad(t, (1, 1, 1, 1, 1, 1)).to(self.dtype)

    def sweep(self, sw, F, vel, axis):
        """One FCT sweep of F along `axis`."""
        d = self.d
        vol = d[0] * d[1] * d[2]
        dvfac = self.dt * d[1] * d[2] if axis == 0 else self.dt * d[0] * d[2] if axis == 1 else self.dt * d[0] * d[1]
        hq, h4 = (d[2], d[2]) if axis == 2 else (d[0], d[1])

        def line(a):  # the sweep axis last, its ghosts kept, those of the other two left out
            return torch.movedim(a, 2 - axis, 2)[1:-1, 1:-1]

        f, uf = line(F), line(vel)[..., 1:]
        FL, FR = f[..., :-1], f[..., 1:]
        ul = uf * self.dt
        lo = sw.pick(uf >= 0, ul * FL, ul * FR)
        hi = sw.pick(uf <= 0, ul * FL, ul * FR)
        a = sw.value(hi - lo)
        dv = vol - dvfac * (uf[..., 1:] - uf[..., :-1])
        df = lo[..., :-1] - lo[..., 1:]
        term = df * d[1] * d[2] / vol if axis == 0 else df * d[1] / (d[0] * d[1]) if axis == 1 else df * d[1] * d[0] / vol
        out = (f[..., 1:-1] + term) * vol / dv
        ftd = sw.pick((out > 1) | (out < 0), self.clamp01(sw, out), out)
        ftd = sw.value(ftd)
        pad = torch.nn.functional.pad(ftd, (1, 1))
        fmx = sw.mx(ftd, sw.mx(pad[..., :-2], pad[..., 2:]))
        fmn = sw.mn(ftd, sw.mn(pad[..., :-2], pad[..., 2:]))
        al, ar = a[..., :-1], a[..., 1:]

        def ratio(plus, minus, q):
            s = sw.value(sw.mx(self.zero, plus) - sw.mn(self.zero, minus))
            some = sw(s > 0)
            r = sw.mn(self.one, q / torch.where(some, s, self.one))
            return torch.nn.functional.pad(torch.where(some, r, self.zero), (1, 1))

        rp, rm = ratio(al, ar, (fmx - ftd) * hq), ratio(ar, al, (ftd - fmn) * hq)
        lim = sw.pick(a >= 0, sw.mn(rp[..., 1:], rm[..., :-1]), sw.mn(rp[..., :-1], rm[..., 1:]))
        lim = torch.cat((torch.zeros_like(lim[..., :1]), lim[..., 1:]), -1)
        ac = a * lim
        out = self.clamp01(sw, ftd - ((ac[..., 1:] - ac[..., :-1]) / h4) * vol / dv)
        F = F.clone()
        torch.movedim(F, 2 - axis, 2)[1:-1, 1:-1, 1:-1] = out
        return F

    def __call__(self, s, istep, sw):
        c, at = self.c, self.at
        F, u, v, w, p = (s[k] for k in STATE)
        rho, nu = self.rho_nu(sw, F)
        star = [sw.value(self.only(self.star(sw, (u, v, w), q, at(nu)), q)) for q in range(3)]
        if c["csf"]:
            kap = self.csf(F)
            for q in range(3):
                m = self._shift(q, -1)
                fa = self.sigma * (0.5 * (at(kap, **m) + at(kap))) * ((at(F) - at(F, **m)) * self.di[q])
                star[q] = self.only(at(star[q]) + self.dt * (fa / (0.5 * (at(rho, **m) + at(rho)))), q)
        rhs = at(rho) / self.dt * ((at(star[0], x=1) - at(star[0])) * self.di[0] +
                                   (at(star[1], y=1) - at(star[1])) * self.di[1] +
                                   (at(star[2], z=1) - at(star[2])) * self.di[2])
        p = self.pressure(p, rhs) if c["mode"] == "plain" else self.solved(rhs)
        p = sw.value(p)
        vel = []
        for q, old in enumerate((u, v, w)):
            m = self._shift(q, -1)
            r = 0.5 * (at(rho) + at(rho, **m))
            new = at(star[q]) - self.dt / r * (at(p) - at(p, **m)) * self.di[q]
            full = old.clone()
            at(full)[...] = at(self.only(new, q))
            vel.append(full)
        vel = [sw.value(x) for x in bc_velocity(*vel)]
        for q in ((0, 1, 2), (1, 2, 0), (2, 0, 1))[istep % 3]:
            F = sw.value(self.sweep(sw, F, vel[q], q))
        F = bc_F(self.clamp01(sw, F))
        return {"F": F, "u": vel[0], "v": vel[1], "w": vel[2], "p": p}


def _exact_adjoint(c, f):
    s32, s64 = _Step(c, torch.float32, f["F"].device), _Step(c, torch.float64, f["F"].device)
    states = [f]
    for n in range(c["steps"]):
        states.append(s32(states[-1], 1 + n, _Plain()))
    b = _box(c)
    centre = [(np.arange(1, n + 1) - 0.5) * float(d) for n, d in zip(s64.n, s64.d)]
    inside = [torch.tensor((x > b[2 * q]) & (x < b[2 * q + 1]), device=f["F"].device) for q, x in enumerate(centre)]
    where = inside[2].view(-1, 1, 1) & inside[1].view(1, -1, 1) & inside[0].view(1, 1, -1)
    dV = float(s64.d[0] * s64.d[1] * s64.d[2])
    last = states[-1]["F"].double()[1:-1, 1:-1, 1:-1]
    loss = float((last * where).sum() * dV)
    lam = {k: torch.zeros_like(f[k], dtype=torch.float64) for k in STATE}
    lam["F"][1:-1, 1:-1, 1:-1] = where * dV
    gg = torch.zeros(3, dtype=torch.float64, device=f["F"].device)
    for n in reversed(range(c["steps"])):
        tape = _Switch()
        s32(states[n], 1 + n, tape)
        x = {k: states[n][k].double().requires_grad_() for k in STATE}
        s64.g = [g.detach().clone().requires_grad_() for g in s64.g]
        y = s64(x, 1 + n, _Switch(tape.out))
        ins = [x[k] for k in STATE] + s64.g
        got = torch.autograd.grad([y[k] for k in STATE], ins, [lam[k] for k in STATE], allow_unused=True)
        got = [torch.zeros_like(i) if g is None else g for i, g in zip(ins, got)]
        lam = dict(zip(STATE, got[:5]))
        gg += torch.stack(got[5:])
        del y, x, got, tape
    return {"loss": loss, "grad_g": gg.cpu().numpy(), "grad": {k: lam[k].cpu().numpy() for k in STATE}}


def exact(case, seed):
    c = dict(case)
    f = _fields(c, seed)
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, f)
    step = _Step(c, torch.float64, f["F"].device)
    dV = float(step.d[0] * step.d[1] * step.d[2])
    s = {k: x.double() for k, x in f.items()}
    f = None
    volumes = []
    for n in range(c["steps"]):
        s = step(s, 1 + n, _Plain())
        volumes.append(float(s["F"][1:-1, 1:-1, 1:-1].sum()) * dV)
    if c["kind"] == "slab":
        return {"state": s, "volume": volumes[-1]}
    if c["host"]:
        s = {k: x.cpu().numpy() for k, x in s.items()}
    if c["volume"] == "none":
        volumes = None
    elif c["volume"] == "async":
        volumes = torch.tensor(volumes, dtype=torch.float64)
    return {"state": s, "volumes": volumes}
