"""What a program has this engine do, as timed cases through its public entry points.

Four kinds of work, each over the range of sizes, storage types and options the
repository's own configurations, tests and benchmark use:

* ``single``: a single-phase culvert channel, advanced and read back.  Periodic
  with a body force (the culvert channel, the 8192x2048 probe), or between an
  inlet and an outlet in the reference's modes, as the file-based set-up runs it.
* ``dam``: a free-surface dam break through a culvert box, the engine's modes or
  the reference's.
* ``batch``: an ensemble of small channels of uneven sizes.
* ``adjoint``: objective and gradient of the porous channel.

A pass continues the case by ``steps`` time steps and reads the results back (into
pinned host memory, as the VTK output takes them, or into device buffers, as a
viewer does); an adjoint pass is one forward and one backward sweep.
"""
import math

import numpy as np
import torch

from flowlb_b200 import cases as C
from flowlb_b200 import engine as E


def listed():
    return [
        # a viewer's loop on the smallest grid of the example inputs (odd sizes): one step per frame
        dict(name="viewer_101x101", kind="single", nx=101, ny=101, precision=32, modes="engine", io=False, steps=1,
             spin=64, host=False),
        # the culvert channel of the single-phase configuration
        dict(name="channel_256x64", kind="single", nx=256, ny=64, precision=32, modes="engine", io=False, steps=200,
             spin=200, host=True),
        # the example inputs' long plane channel between an inlet and an outlet, in the reference's modes
        dict(name="inlet_channel_4001x41", kind="single", nx=4001, ny=41, precision=32, modes="reference", io=True,
             steps=200, spin=200, host=True),
        # a ragged mid-size channel in double precision
        dict(name="channel_1023x255_f64", kind="single", nx=1023, ny=255, precision=64, modes="engine", io=False,
             steps=100, spin=100, host=True),
        # the bandwidth probe, in single precision and with FP16 storage
        dict(name="channel_8192x2048", kind="single", nx=8192, ny=2048, precision=32, modes="engine", io=False,
             steps=100, spin=20, host=False),
        dict(name="channel_8192x2048_f16", kind="single", nx=8192, ny=2048, precision=16, modes="engine", io=False,
             steps=100, spin=20, host=False),
        # the benchmark's dam break, and the storage sweep's
        dict(name="dam_2048x512", kind="dam", nx=2048, ny=512, precision=32, modes="engine", steps=200, spin=400,
             host=True),
        dict(name="dam_8192x2048", kind="dam", nx=8192, ny=2048, precision=32, modes="engine", steps=50, spin=100,
             host=False),
        # the example inputs' small dam break: reference modes, subgrid model, FP32 mass
        dict(name="dam_101x101_reference", kind="dam", nx=101, ny=101, precision=32, modes="reference", steps=50,
             spin=50, host=True),
        # part of the culvert ensemble, in the form its autotuner picks for many cases
        dict(name="batch_48_streams", kind="batch", cases=48, form="streams", steps=200, spin=0),
        # the outlet-discharge gradient, double precision; and a ragged one in single precision
        dict(name="adjoint_1024x256_f64", kind="adjoint", nx=1024, ny=256, precision=64, steps=512, window=64, every=64),
        dict(name="adjoint_517x131_f32", kind="adjoint", nx=517, ny=131, precision=32, steps=256, window=64, every=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "dam", "dam", "batch", "adjoint"])
    if kind == "single":
        nx, ny = _log(rng, 96, 8192), _log(rng, 40, 2048)
        if rng.random() < 0.5:
            nx = max(96, nx // 8 * 8)  # half of them rows of whole vectors
        modes = rng.choice(["engine", "engine", "reference"])
        precision = rng.choice([32, 32, 16, 64])
        if precision == 64 or modes == "reference":
            ny = max(40, ny // 2)  # dearer per cell
        return dict(kind=kind, nx=nx, ny=ny, precision=precision, modes=modes,
                    io=modes == "reference" and rng.random() < 0.5, steps=rng.choice([1, 20, 100]), spin=40,
                    host=nx * ny < 1 << 20)
    if kind == "dam":
        nx = _log(rng, 96, 4096)
        ny = max(64, int(nx * rng.uniform(0.2, 0.6)))
        modes = rng.choice(["engine", "engine", "reference"])
        return dict(kind=kind, nx=nx, ny=ny, precision=32 if modes == "reference" else rng.choice([32, 32, 16, 64]),
                    modes=modes, steps=40, spin=rng.choice([20, 100]), host=nx * ny < 1 << 20)
    if kind == "batch":
        return dict(kind=kind, cases=_log(rng, 4, 48), form=rng.choice(["streams", "streams", "cluster"]),
                    steps=rng.choice([100, 200]), spin=0)
    nx, ny = _log(rng, 96, 1024), _log(rng, 48, 256)
    return dict(kind=kind, nx=nx, ny=ny, precision=rng.choice([32, 64]), steps=128, window=rng.choice([32, 128]),
                every=rng.choice([16, 32, 64]))


# ---- the cases' inputs -----------------------------------------------------------


def _single_inputs(case, seed):
    """Geometry and parameters of a single-phase case: a seed-placed culvert block, tau and force."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    w = max(2, int(rng.uniform(0.05, 0.2) * nx))
    h = max(1, int(rng.uniform(0.2, 0.5) * ny))
    x0 = int(rng.uniform(0.3, 0.6) * nx)
    flags = C.channel_with_block(nx, ny, x0, x0 + w, min(ny - 2, 1 + h))
    tau = float(np.float32(rng.uniform(0.55, 0.8)))
    # a velocity of a few hundredths: in the channel's steady profile, or after 10,000 steps on the largest grids
    g = max(8.0 * (tau - 0.5) / 3.0 / ny ** 2, 1e-4 if nx * ny >= 1 << 22 else 0.0)
    p = dict(tau=tau, fx=float(np.float32(rng.uniform(0.02, 0.08) * g)), fy=0.0)
    if case["io"]:
        flags[1:ny - 1, 0] = C.INLET
        flags[1:ny - 1, nx - 1] = C.OUTLET
        p.update(inlet_ux=float(rng.uniform(0.02, 0.05)), inlet_uy=0.0)
    return flags, p


def _dam_inputs(case, seed):
    """A water column beside a culvert box in a walled tank, sizes moved a little by the seed."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    flags = np.full((ny, nx), C.GAS, np.uint8)
    flags[0, :] = flags[ny - 1, :] = C.WALL
    flags[:, 0] = flags[:, nx - 1] = C.WALL
    flags[1:int(rng.uniform(0.57, 0.63) * ny), 1:int(rng.uniform(0.38, 0.42) * nx)] = C.FLUID
    box, top, opening = max(4, nx // 8), max(6, int(0.31 * ny)), max(3, int(0.19 * ny))
    cx = int(rng.uniform(0.56, 0.62) * nx)
    flags[1 + opening:1 + top, cx - box // 2:cx + box // 2] = C.WALL
    p = dict(tau=float(np.float32(rng.uniform(0.55, 0.57))), fx=0.0, fy=-float(np.float32(rng.uniform(4e-5, 6e-5))))
    return flags, p


def _modes(case):
    """Engine defaults, or the reference's modes as flb_setup_from_files selects them."""
    if case["modes"] == "reference":
        m = dict(bounce_back=E.BB_IMPLICIT, arithmetic=E.ARITH_REFERENCE)
        if case["kind"] == "dam":
            m.update(fs_mode=E.FS_REFERENCE, mass_precision=32, subgrid=True, u_max=0.25)
        return m
    m = dict(bounce_back=E.BB_HALFWAY, arithmetic=E.ARITH_FUSED)
    if case["kind"] == "dam":
        m.update(fs_mode=E.FS_CONSERVATIVE, u_max=0.25)
    return m


def _batch_inputs(case, seed):
    """The culvert ensemble's geometries, with the seed's relaxation times and forces (as the ensemble draws them, the
    force limited so that no case's steady velocity leaves the model's range)."""
    rng = np.random.default_rng(seed)
    out = []
    for c in C.ensemble(case["cases"]):
        tau = float(np.float32(rng.uniform(0.52, 0.8)))
        gx = min(10.0 ** rng.uniform(-7.0, -5.0), 0.8 * (tau - 0.5) / 3.0 / c.ny ** 2)
        out.append((c.flags, tau, float(np.float32(gx)), 0.0))
    return out


def _adjoint_inputs(case, seed):
    c = C.porous_channel(case["nx"], case["ny"], seed=seed)
    return c.flags, c.porosity.astype(np.float64), dict(tau=0.6, gx=float(np.random.default_rng(seed).uniform(4e-6, 6e-6)))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = E.Batch(_batch_inputs(case, seed), autotune=0)
        if case["form"] == "streams":
            b.set_launch("streams", 1, min(16, case["cases"]), 0)
        return dict(case=case, batch=b)
    if kind == "adjoint":
        flags, s, p = _adjoint_inputs(case, seed)
        return dict(case=case, adjoint=E.Adjoint(flags, s, precision=case["precision"], steps=case["steps"],
                                                 window=case["window"], checkpoint_every=case["every"], **p))
    flags, p = (_single_inputs if kind == "single" else _dam_inputs)(case, seed)
    solver = E.Solver(flags, free_surface=kind == "dam", precision=case["precision"], **p, **_modes(case))
    solver.step(case["spin"])
    solver.sync()
    fields = [("rho", E.FIELD_RHO), ("u", E.FIELD_U)]
    if kind == "dam":
        fields += [("phi", E.FIELD_PHI), ("flags", E.FIELD_FLAGS)]
    out = {}
    for name, fid in fields:
        size, count = solver.field_info(fid)
        dt = {1: torch.uint8, 4: torch.float32, 8: torch.float64}[size]
        out[name] = (torch.empty(count, dtype=dt, pin_memory=True) if case["host"]
                     else torch.empty(count, dtype=dt, device="cuda"))
    return dict(case=case, solver=solver, fields=fields, out=out)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        b.sync()
        return [b.read(i, E.FIELD_U) for i in range(b.n)]
    if case["kind"] == "adjoint":
        a = state["adjoint"]
        J = a.forward()
        ds, dg = a.backward()
        return dict(J=J, ds=ds, dg=dg)
    s, out = state["solver"], state["out"]
    s.step(case["steps"])
    for name, fid in state["fields"]:
        if case["host"]:
            s.read(fid, out[name].numpy())
        else:
            s.read_device(fid, out[name].data_ptr())
    return out


def work(case):
    """Bytes: the state (nine populations per cell, and the free surface's mass, excess, fill level and flag)
    read and written once per pass, and the results.  Flops: a D2Q9 collision is about 110 operations per cell and
    step; the free surface adds about as many again on its cells (about a quarter of the tank); the adjoint's
    reverse step about 200, with one recomputation."""
    kind = case["kind"]
    if kind == "batch":
        cells = sum(f.size for f, *_ in _batch_inputs(case, 1))
        return dict(bytes=cells * (72.0 + 8.0), flops=110.0 * cells * case["steps"])
    cells, c = case["nx"] * case["ny"], case["precision"] / 8.0
    if kind == "adjoint":
        segments = case["steps"] // case["every"]
        return dict(bytes=cells * (2.0 * 9.0 * c * segments + 8.0 + 8.0), flops=420.0 * cells * case["steps"])
    out = 8.0 if c == 8 else 4.0
    if kind == "single":
        return dict(bytes=cells * (18.0 * c + 3.0 * out), flops=110.0 * cells * case["steps"])
    m = 4.0 if case["modes"] == "reference" else 8.0
    live = 0.25 * cells
    return dict(bytes=live * (18.0 * c + 6.0 * m + 2.0) + cells * (3.0 * out + m + 1.0), flops=220.0 * live * case["steps"])


# ---- the same model in 64 bits ---------------------------------------------------

_CX = [0, 1, -1, 0, 0, 1, -1, 1, -1]
_CY = [0, 0, 0, 1, -1, 1, -1, -1, 1]
_W = [4.0 / 9.0] + [1.0 / 9.0] * 4 + [1.0 / 36.0] * 4


def _to(a, i):
    """The values at c + e_i, for every cell c (periodic)."""
    return torch.roll(a, (-_CY[i], -_CX[i]), (0, 1))


def _from(a, i):
    """The values at c - e_i."""
    return torch.roll(a, (_CY[i], _CX[i]), (0, 1))


def _equilibrium(rho, ux, uy):
    usq = 1.5 * (ux * ux + uy * uy)
    out = []
    for i in range(9):
        cu = _CX[i] * ux + _CY[i] * uy
        out.append(_W[i] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq))
    return out


def _limit(ux, uy, umax):
    if umax <= 0.0:
        return ux, uy
    n = torch.sqrt(ux * ux + uy * uy)
    k = torch.where(n > umax, umax / n.clamp_min(1e-300), torch.ones_like(n))
    return ux * k, uy * k


def _moments(f):
    rho = sum(f)
    return rho, (f[1] - f[2] + f[5] - f[6] + f[7] - f[8]) / rho, (f[3] - f[4] + f[5] - f[6] + f[8] - f[7]) / rho


class _Model:
    """The D2Q9 step on (ny, nx) float64 tensors.  Populations sit in nine link slots: at a step of parity q the pair
    (i, i + 1), i odd, of a cell is read from its own slot a and the slot b of the cell toward i, and written back the
    other way round, so a link into a cell that is not updated keeps what was sent into it."""

    def __init__(self, flags, p, modes, free_surface):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        g = torch.from_numpy(flags.astype(np.int64)).to(dev)
        self.om, self.fx, self.fy = 1.0 / p["tau"], p["fx"], p["fy"]
        self.hw = modes["bounce_back"] == E.BB_HALFWAY
        self.cons = modes.get("fs_mode", E.FS_CONSERVATIVE) == E.FS_CONSERVATIVE
        self.subgrid, self.umax, self.fs = modes.get("subgrid", False), modes.get("u_max", 0.0), free_surface
        self.wall = (g & C.WALL) != 0
        self.inlet, self.outlet = (g & C.INLET) != 0, (g & C.OUTLET) != 0
        self.io = bool((self.inlet | self.outlet).any())
        zero = torch.zeros(g.shape, dtype=torch.float64, device=dev)
        self.rho = zero + 1.0
        self.ux = torch.where(self.inlet, zero + p.get("inlet_ux", 0.0), zero)
        self.uy = torch.where(self.inlet, zero + p.get("inlet_uy", 0.0), zero)
        self.flags, self.t = g, 0
        self.F = [zero.clone() for _ in range(9)]
        self._store(_equilibrium(self.rho, self.ux, self.uy), ~self.wall if self.hw else ~torch.zeros_like(self.wall), 1)
        if free_surface:
            fluid = g == C.FLUID
            ny, nx = g.shape
            near, early = torch.zeros_like(fluid), torch.zeros_like(fluid)
            for i in range(1, 9):
                n = _to(fluid, i)  # the tank's frame is wall: no fluid wraps around
                near |= n
                if _CY[i] < 0 or (_CY[i] == 0 and _CX[i] < 0):
                    early |= n
            new = (g == C.GAS) & near
            self.flags = torch.where(new, torch.full_like(g, C.INTERFACE), g)
            self.mass = fluid.double() + 0.5 * (new & early).double()
            self.phi, self.excess = self.mass.clone(), zero.clone()

    @staticmethod
    def _slots(i, odd):
        return (i, i + 1) if odd else (i + 1, i)

    def _load(self, odd):
        F, f = self.F, [self.F[0]] + [None] * 8
        for i in (1, 3, 5, 7):
            a, b = self._slots(i, odd)
            f[i], f[i + 1] = F[a], _to(F[b], i)
            if self.hw:
                f[i] = torch.where(_from(self.wall, i), F[b], f[i])
                f[i + 1] = torch.where(_to(self.wall, i), _to(F[a], i), f[i + 1])
        return f

    def _store(self, f, act, odd):
        F = self.F
        F[0] = torch.where(act, f[0], F[0])
        for i in (1, 3, 5, 7):
            a, b = self._slots(i, odd)
            F[b] = torch.where(_from(act, i), _from(f[i], i), F[b])
            F[a] = torch.where(act, f[i + 1], F[a])

    def _fs1(self, odd):
        """Mass exchange over the links, and the populations an interface cell rebuilds toward gas."""
        F, flags = self.F, self.flags
        e = flags & 7
        act = (e == C.FLUID) | (e == C.INTERFACE)
        if self.cons:
            act &= (flags & C.WALL) == 0
        f = self._load(odd)
        out = [f[0]] + [None] * 8
        for i in (1, 3, 5, 7):
            a, b = self._slots(i, odd)
            out[i], out[i + 1] = _to(F[a], i), F[b]
        m = self.mass + sum(_to(self.excess, i) for i in range(1, 9))
        rho, ux, uy = _moments(out)
        phi0 = self.phi if self.cons else self._fill(m, rho)
        opp = [0, 2, 1, 4, 3, 6, 5, 8, 7]
        add = torch.zeros_like(m)
        for i in range(1, 9):
            ne = _to(e, i)
            d = f[opp[i]] - out[i]
            mixed = ((ne == C.FLUID).double() + (ne == C.INTERFACE).double() * 0.5 * (_to(self.phi, i) + phi0)) * d
            plain = d if not self.cons else d * ((ne == C.FLUID) | (ne == C.INTERFACE)).double()
            add = add + torch.where(e == C.FLUID, plain, mixed)
        ux, uy = _limit(ux + 0.5 * self.fx / rho, uy + 0.5 * self.fy / rho, self.umax)
        feq = _equilibrium(torch.ones_like(rho), ux, uy)
        surf = act & (e == C.INTERFACE)
        for i in range(1, 9):
            # rebuilt where the population arrives from gas (conservative), or travels toward it (reference)
            gas = _to(e, opp[i] if self.cons else i) == C.GAS
            f[i] = torch.where(surf & gas, feq[i] - out[opp[i]] + feq[opp[i]], f[i])
        self.mass = torch.where(act, m + add, self.mass)
        return f

    @staticmethod
    def _fill(m, rho):
        return torch.where(rho > 0, (m / rho).clamp(0.0, 1.0), torch.full_like(m, 0.5))

    def _flag_pass(self, odd):
        fl, f0 = self.flags, self.flags
        solid = (f0 & (C.WALL | C.MOVING_WALL | C.INLET)) != 0

        def near(mask):
            r = torch.zeros_like(mask)
            for i in range(1, 9):
                r |= _to(mask, i)
            return r

        any_if = near((fl & 5) == 5)
        fl = torch.where(any_if & ((f0 & 6) == 6), fl & ~C.GAS, fl)
        fl = torch.where(any_if & ((f0 & 6) == C.GAS), (fl & ~C.GAS) | C.GAS_INTERFACE, fl)
        f1 = fl
        any_ig = near((f1 & 0x86) == 6)
        back = any_ig & (((f1 & 0x25) == C.FLUID) | ((f1 & 0x25) == 5))
        fl = torch.where(back, (fl & ~5) | C.INTERFACE, fl)
        born = (f1 & 0x86) == C.GAS_INTERFACE
        if bool(born.any()):
            wet = ((f1 & 5) != 0).double()
            n = sum(_to(wet, i) for i in range(1, 9))
            avg = [torch.where(n > 0, sum(_to(wet * q, i) for i in range(1, 9)) / n.clamp_min(1.0), torch.zeros_like(n))
                   for q in (self.rho, self.ux, self.uy)]
            r = torch.where(born, avg[0], torch.ones_like(n))
            ux, uy = _limit(avg[1] + 0.5 * self.fx / r, avg[2] + 0.5 * self.fy / r, self.umax)
            self._store(_equilibrium(avg[0], ux, uy), born, odd)
        sw = fl & 0x87
        f3 = fl
        to_plain = ~solid & ((sw == 5) | (sw == 6))
        fl = torch.where(to_plain, fl & ~C.INTERFACE, fl)
        fl = torch.where(~solid & (sw == C.GAS_INTERFACE), (fl & ~C.GAS_INTERFACE) | C.INTERFACE, fl)
        if self.cons:
            wet = (((fl & 7) == C.FLUID) | ((fl & 7) == C.INTERFACE)) & ~solid
        else:
            wet = ((((f3 & C.FLUID) != 0) | ((fl & C.INTERFACE) != 0)) != ((fl & C.GAS_INTERFACE) != 0))
        n = sum(_to(wet.double(), i) for i in range(1, 9))
        m, rho, zero = self.mass, self.rho, torch.zeros_like(self.mass)
        full, empty, part = (sw == 1) | (sw == 5), (sw == 2) | (sw == 6), (sw == 4) | (sw == 128)
        over, under = part & (m > rho), part & (m < 0) & ~(m > rho)
        ex = torch.where(full | over, m - rho, torch.where(empty | under, m, zero))
        m2 = torch.where(full | over, rho, torch.where(empty | under, zero, m))
        ph = torch.where(full, zero + 1.0, torch.where(part, self._fill(m2, rho), zero))
        m2 = m2 + torch.where(n > 0, zero, ex)
        ex = torch.where(n > 0, ex / n.clamp_min(1.0), zero)
        self.mass = torch.where(solid, self.mass, m2)
        self.excess = torch.where(solid, self.excess, ex)
        self.phi = torch.where(solid, self.phi, ph)
        self.flags = fl

    def step(self):
        odd = self.t & 1
        flags = self.flags
        act = (flags & (C.GAS | C.WALL)) == 0
        f = self._fs1(odd) if self.fs else self._load(odd)
        rho, ux, uy = _moments(f)
        if self.io:
            flat = lambda q, d: torch.roll(q.reshape(-1), d).reshape(q.shape)  # noqa: E731
            r0, x0, y0 = self.rho, self.ux, self.uy
            rho = torch.where(self.inlet, flat(r0, -1), torch.where(self.outlet, r0, rho))
            ux = torch.where(self.inlet, x0, torch.where(self.outlet, flat(x0, 1), ux))
            uy = torch.where(self.inlet, y0, torch.where(self.outlet, flat(y0, 1), uy))
        if self.fs:
            e = flags & 7
            no_fluid, no_gas = torch.ones_like(act), torch.ones_like(act)
            for i in range(1, 9):
                ne = _to(e, i)
                no_fluid &= ne != C.FLUID
                no_gas &= ne != C.GAS
            surf = act & ((flags & C.INTERFACE) != 0)
            up = surf & ((self.mass > 1.001 * rho) | no_gas)
            down = surf & ~up & ((self.mass < -0.001) | no_fluid)
            flags = torch.where(up, (flags & ~7) | 5, torch.where(down, (flags & ~7) | 6, flags))
        ux, uy = _limit(ux + 0.5 * self.fx / rho, uy + 0.5 * self.fy / rho, self.umax)
        keep_u = act & ~self.inlet
        self.rho = torch.where(act, rho, self.rho)
        self.ux, self.uy = torch.where(keep_u, ux, self.ux), torch.where(keep_u, uy, self.uy)
        feq = _equilibrium(rho, ux, uy)
        om = torch.full_like(rho, self.om)
        if self.subgrid:
            d = [f[i] - feq[i] for i in range(9)]
            hxx = sum(_CX[i] ** 2 * d[i] for i in range(1, 9))
            hyy = sum(_CY[i] ** 2 * d[i] for i in range(1, 9))
            hxy = sum(_CX[i] * _CY[i] * d[i] for i in range(1, 9))
            q = hxx * hxx + hyy * hyy + 2.0 * hxy * hxy
            tau = 1.0 / om
            om = 2.0 / (tau + torch.sqrt(tau * tau + 0.54037965 * torch.sqrt(q) / rho))
        uf = ux * self.fx + uy * self.fy
        set_eq = self.inlet | self.outlet
        post = []
        for i in range(9):
            cf, cu = _CX[i] * self.fx + _CY[i] * self.fy, _CX[i] * ux + _CY[i] * uy
            force = _W[i] * (3.0 * (cf - uf) + 9.0 * cu * cf)
            v = f[i] + om * (feq[i] - f[i]) + (1.0 - 0.5 * om) * force
            post.append(torch.where(set_eq, feq[i], v) if self.io else v)
        self._store(post, act, odd)
        self.flags = flags
        if self.fs:
            self._flag_pass(odd)
        self.t += 1


def _exact_solver(case, seed):
    flags, p = (_single_inputs if case["kind"] == "single" else _dam_inputs)(case, seed)
    m = _Model(flags, p, _modes(case), case["kind"] == "dam")
    for _ in range(case["spin"] + case["steps"]):
        m.step()
    out = dict(rho=m.rho.reshape(-1), u=torch.cat([m.ux.reshape(-1), m.uy.reshape(-1)]))
    if case["kind"] == "dam":
        out.update(phi=m.phi.reshape(-1), flags=None)
    return out


def _exact_batch(case, seed):
    out = []
    for flags, tau, fx, fy in _batch_inputs(case, seed):
        m = _Model(flags, dict(tau=tau, fx=fx, fy=fy), dict(bounce_back=E.BB_HALFWAY), False)
        for _ in range(case["steps"]):
            m.step()
        out.append(torch.cat([m.ux.reshape(-1), m.uy.reshape(-1)]))
    return out


def _exact_adjoint(case, seed):
    """The objective and its gradient by reverse-mode differentiation of the whole run, a segment at a time."""
    flags, s, p = _adjoint_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    wall = torch.from_numpy(flags == C.WALL).to(dev)
    s = torch.from_numpy(s).to(dev).requires_grad_()
    g = torch.tensor([p["gx"], 0.0], dtype=torch.float64, device=dev, requires_grad=True)
    om, steps, window = 1.0 / p["tau"], case["steps"], case["window"]
    opp = [0, 2, 1, 4, 3, 6, 5, 8, 7]
    from_wall = [_from(wall, i) for i in range(9)]

    def segment(state, t0, n):
        post, J = list(state), torch.zeros((), dtype=torch.float64, device=dev)
        for t in range(t0, t0 + n):
            f = [post[0]] + [torch.where(from_wall[i], post[opp[i]], _from(post[i], i)) for i in range(1, 9)]
            rho, vx, vy = _moments(f)
            ux, uy = (vx + 0.5 * g[0]) / (1.0 + 0.5 * s), (vy + 0.5 * g[1]) / (1.0 + 0.5 * s)
            fx, fy = rho * (g[0] - s * ux), rho * (g[1] - s * uy)
            feq, uf = _equilibrium(rho, ux, uy), ux * fx + uy * fy
            new = []
            for i in range(9):
                cf, cu = _CX[i] * fx + _CY[i] * fy, _CX[i] * ux + _CY[i] * uy
                force = _W[i] * (3.0 * (cf - uf) + 9.0 * cu * cf)
                new.append(torch.where(wall, post[i], (1.0 - om) * f[i] + om * feq[i] + (1.0 - 0.5 * om) * force))
            post = new
            if t + window >= steps:
                J = J + torch.where(wall, torch.zeros_like(rho), rho * ux)[:, -1].sum() / window
        return post, J

    n, rest = 16, torch.ones(flags.shape, dtype=torch.float64, device=dev)
    states, J = [[w * rest for w in _W]], 0.0
    with torch.no_grad():
        for t in range(0, steps, n):
            nxt, j = segment(states[-1], t, min(n, steps - t))
            J += float(j)
            states.append(nxt)
    lam = [torch.zeros_like(rest) for _ in range(9)]
    for k in range(len(states) - 2, -1, -1):
        inp = [v.detach().requires_grad_() for v in states[k]]
        nxt, j = segment(inp, k * n, min(n, steps - k * n))
        total = j + sum((a * b).sum() for a, b in zip(nxt, lam))
        total.backward()
        lam = [v.grad for v in inp]
    return dict(J=J, ds=s.grad, dg=g.grad)


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        return _exact_batch(case, seed) if case["kind"] == "batch" else _exact_solver(case, seed)
