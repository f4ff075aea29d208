"""Work that programs using nmhd_b200 have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (the solver, its initial state, result buffers), ``run`` is
one pass through the public entry points, ``exact`` the same results in 64
bits from a plain torch restatement of the scheme.

Kinds of case:

``box``       MHDSolver on device states: set the state and the clock, take
              ``steps`` steps, read the state and the clock.  Every pass starts
              from the same state, so passes are alike.
``monitored`` MHDSolver with a monitor() that takes the diagnostics before
              every step, as the reference's applications do.
``slabs``     SlabGroup: one box as radial slabs in one process.
``ensemble``  BatchSolver on host states: set every state, steps, read every
              state (the batch's clock runs on from pass to pass).
``adjoint``   MHDSolver.adjoint: the loss and its gradient with respect to the
              initial state.
"""
import math

import numpy as np
import torch

from nmhd_b200.batch import BatchSolver
from nmhd_b200.config import FLAG_FAST_ARITHMETIC, SolverConfig
from nmhd_b200.slab import SlabGroup, slab_config
from nmhd_b200.solver import MHDSolver

GAMMA = 5.0 / 3.0
FIELDS = ("density", "vx", "vy", "vz", "pressure", "bx", "by", "bz")


def _box(kind, problem, nx, ny, nz, steps, **more):
    """nx azimuthal (x), ny radial (y), nz vertical (z) interior cells."""
    case = dict(kind=kind, problem=problem, nx=nx, ny=ny, nz=nz, steps=steps, lx=1.0, ly=1.0, lz=1.0, my=0, mz=0,
                space_order=2, time_order=2, fast=False, start="developed", beta=400.0, q=1.5)
    if problem == "shearing_box":
        case.update(my=4, lx=4.0)
    case.update(more)
    return case


def listed():
    cases = [
        # the smallest calls: launches and latency are all there is
        ("vortex_16", _box("box", "vortex", 16, 16, 16, 16)),
        # a monitored run: one step per call, diagnostics before each
        ("monitored_64x32x32", _box("monitored", "shearing_box", 64, 32, 32, 4)),
        # the 64^3 Orszag-Tang vortex
        ("vortex_64", _box("box", "vortex", 64, 64, 64, 16)),
        # odd sizes, spacings that are no powers of two, margins in y and z
        ("ragged_250x97x61", _box("box", "shearing_box", 250, 97, 61, 8, mz=3, my=3, lx=2.5, lz=0.6)),
        # the MRI shearing box of the benchmark, from its quiet start
        ("mri_256x128x64", _box("box", "shearing_box", 256, 128, 64, 16, start="quiet")),
        # the same box with the opt-in fast arithmetic
        ("fast_256x128x64", _box("box", "shearing_box", 256, 128, 64, 16, start="quiet", fast=True)),
        # the 256^3 vortex
        ("vortex_256", _box("box", "vortex", 256, 256, 256, 4)),
        # the largest box of the benchmark
        ("mri_1024x512x256", _box("box", "shearing_box", 1024, 512, 256, 2)),
        # one box as two radial slabs, launched step by step
        ("slabs_2x256x64x64", _box("slabs", "shearing_box", 256, 128, 64, 8, slabs=2)),
        # an ensemble of uneven boxes (sides 32 to 96), host states in and out
        ("ensemble_12", dict(kind="ensemble", boxes=12, low=32, high=96, steps=8)),
        # many small boxes (sides 8 to 16)
        ("ensemble_small_256", dict(kind="ensemble", boxes=256, low=8, high=16, steps=16)),
        # gradient of the Maxwell stress on the 64^3 shearing box
        ("adjoint_64", _box("adjoint", "shearing_box", 64, 64, 64, 20, lx=1.0, ckpt=10, budget=-1)),
    ]
    return [dict(case, name=name) for name, case in cases]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["box"] * 6 + ["monitored", "slabs", "ensemble", "ensemble", "adjoint", "adjoint"])
    if kind == "ensemble":
        if rng.random() < 0.5:
            return dict(kind=kind, boxes=rng.randint(3, 12), low=rng.randint(24, 40), high=rng.randint(48, 96),
                        steps=rng.choice([2, 4, 8]))
        return dict(kind=kind, boxes=rng.randint(40, 256), low=rng.randint(8, 10), high=rng.randint(12, 20),
                    steps=rng.choice([4, 8, 16]))
    top = {"box": 512, "monitored": 96, "slabs": 192, "adjoint": 72}[kind]
    shearing = kind == "slabs" or rng.random() < 0.6
    nx, ny, nz = _log(rng, 16, top), _log(rng, 12, top // 2), _log(rng, 8, top // 2)
    if rng.random() < 0.5:  # rows of whole 16-byte chunks
        nx = max(8, nx // 8 * 8)
    cells = nx * ny * nz
    more = dict(lx=round(rng.uniform(0.5, 4.0), 3), ly=round(rng.uniform(0.5, 2.0), 3), lz=round(rng.uniform(0.5, 2.0), 3),
                start=rng.choice(["developed", "developed", "quiet"]), beta=round(10.0 ** rng.uniform(2.0, 4.0), 2),
                q=round(rng.uniform(1.2, 1.8), 3))
    if shearing and kind != "slabs" and rng.random() < 0.25:
        more["mz"] = rng.randint(2, 4)
    if shearing:
        more["my"] = rng.randint(3, 4)
    if kind == "box":
        if rng.random() < 0.15:
            more[rng.choice(["space_order", "time_order"])] = 1
        elif rng.random() < 0.12:
            more["fast"] = True
    steps = max(1, min(16, int(4e7 / cells)))
    if kind == "slabs":
        more["slabs"] = rng.choice([2, 3, 4])
        ny = max(6, ny // more["slabs"]) * more["slabs"]
        steps = min(steps, 8)
    if kind == "monitored":
        steps = rng.randint(1, 6)
    if kind == "adjoint":
        steps = max(4, min(24, int(6e6 / cells)))
        more.update(ckpt=rng.choice([3, 5, 10]), budget=rng.choice([-1, 0]))
    return _box(kind, "shearing_box" if shearing else "vortex", nx, ny, nz, steps, **more)


# ---------------------------------------------------------------------------
# Configurations and initial states


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _config(c):
    return SolverConfig(size_x=c["nx"], size_y=c["ny"] + 2 * c["my"], size_z=c["nz"] + 2 * c["mz"], margin_y=c["my"],
                        margin_z=c["mz"], extent_x=c["lx"], extent_y=c["ly"], extent_z=c["lz"], gamma=GAMMA, cfl=0.4,
                        problem="shearing_box" if c["problem"] == "shearing_box" else "none", q=c["q"], omega=1.0,
                        space_order=c["space_order"], time_order=c["time_order"],
                        flags=FLAG_FAST_ARITHMETIC if c["fast"] else 0)


def _boxes(c, seed):
    """The boxes of an ensemble case: sizes, field strengths and shears from the case, noise from the seed."""
    r = np.random.Generator(np.random.PCG64(c["boxes"] + 1000 * c["low"] + 100000 * c["high"]))
    sides = np.linspace(c["low"], c["high"], 4 if c["high"] >= 48 else 3).round().astype(int)
    out = []
    for b in range(c["boxes"]):
        n, nz, k = int(r.choice(sides)), int(r.choice(sides)), int(r.choice([2, 3, 4]))
        out.append((_box("box", "shearing_box", k * n, n, nz, c["steps"], lx=float(k), start="quiet",
                         beta=float(10.0 ** r.uniform(2.0, 4.0)), q=float(r.uniform(1.2, 1.8))), seed * 4099 + b))
    return out


def _spacing(length, interior, size):
    """Cell size and padded extent, in float32 steps as the solver derives them."""
    extent = np.float32(length) / np.float32(interior) * np.float32(size)
    return float(extent / np.float32(size)), float(extent)


def _geometry(c, slabs=1):
    """Spacings, the radial coordinate's origin and the velocity across the box of one slab."""
    rows = c["ny"] // slabs
    dx, ex = _spacing(c["lx"], c["nx"], c["nx"])
    dy, ey = _spacing(c["ly"], c["ny"], rows + 2 * c["my"])
    dz, _ = _spacing(c["lz"], c["nz"], c["nz"] + 2 * c["mz"])
    shear = c["problem"] == "shearing_box"
    q, rows_extent = float(np.float32(c["q"])), float(np.float32(c["ly"]) / np.float32(c["ny"]) * np.float32(rows))
    return dict(dx=dx, dy=dy, dz=dz, extent_x=ex, corner_y=-ey / 2, rel_vel=-q * rows_extent if shear else 0.0, q=q,
                omega=1.0, gamma=float(np.float32(GAMMA)), cfl=float(np.float32(0.4)), shear=shear, my=c["my"], mz=c["mz"],
                order2=c["space_order"] == 2, midpoint=c["time_order"] == 2)


def _waves(out, x, y, z, length, rng, amplitude):
    """Adds four random standing waves with the box's periods to `out` at the coordinates x, y, z."""
    dev = out.device
    for _ in range(4):
        f = []
        for at, span in ((z, length[2]), (y, length[1]), (x, length[0])):
            k = 2 * math.pi * int(rng.integers(1, 4)) / span
            f.append(torch.from_numpy(np.cos(k * at + rng.uniform(0, 2 * math.pi)).astype(np.float32)).to(dev))
        out += (amplitude / 2 * f[0])[:, None, None] * f[1][None, :, None] * f[2][None, None, :]
    return out


def _state(c, seed, slab=0, slabs=1):
    """An initial state (8, Sz, Sy, Sx) float32 on the device; the state of radial slab `slab` where there are several."""
    dev, geo = _device(), _geometry(c, slabs)
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=dev).manual_seed(seed * slabs + slab)
    rows, my, mz = c["ny"] // slabs, c["my"], c["mz"]
    shape = (c["nz"] + 2 * mz, rows + 2 * my, c["nx"])
    length = (c["lx"], c["ly"], c["lz"])
    d = (geo["dx"], geo["dy"], geo["dz"])
    lower = [np.arange(shape[2]) * d[0], (np.arange(shape[1]) - my + slab * rows) * d[1], (np.arange(shape[0]) - mz) * d[2]]
    mid = [at + 0.5 * h for at, h in zip(lower, d)]
    w = torch.zeros((8,) + shape, device=dev)
    if c["problem"] == "vortex":
        k = [2 * math.pi / s for s in length]
        ph = rng.uniform(0, 2 * math.pi, 5)
        b0 = 1 / math.sqrt(4 * math.pi)

        def row(v, axis):
            v = torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).to(dev)
            return v.reshape([-1 if a == axis else 1 for a in range(3)])
        w[0], w[4] = 25 / (36 * math.pi), 5 / (12 * math.pi)
        w[1] = -row(np.sin(k[1] * mid[1] + ph[0]), 1)
        w[2] = row(np.sin(k[0] * mid[0] + ph[1]), 2)
        w[3] = 0.1 * row(np.sin(k[2] * mid[2] + ph[2]), 0)
        # differences of the vector potential B0 (cos(ky y) / ky + cos(2 kx x) / (2 kx)) along the edges
        az_y = b0 * np.cos(k[1] * np.append(lower[1], lower[1][-1] + d[1]) + ph[3]) / k[1]
        az_x = b0 * np.cos(2 * k[0] * np.append(lower[0], lower[0][-1] + d[0]) + ph[4]) / (2 * k[0])
        w[5] = row(np.diff(az_y) / d[1], 1)
        w[6] = row(-np.diff(az_x) / d[0], 2)
        w[7] = 0.3 * b0 * row(np.cos(k[0] * mid[0] + ph[1]), 2)
        return w
    w[0], w[4] = 1.0, 1.0
    w[1] = torch.from_numpy((-geo["q"] * (geo["corner_y"] + d[1] * (np.arange(shape[1]) + 0.5))).astype(np.float32)).to(
        dev)[None, :, None]
    w[7] = math.sqrt(2.0 / c["beta"])
    cs = math.sqrt(GAMMA)
    if c["start"] == "developed":
        _waves(w[0], *mid, length, rng, 0.1)
        _waves(w[4], *mid, length, rng, 0.1)
        for v in (1, 2, 3):
            _waves(w[v], *mid, length, rng, 0.1 * cs)
        # B += curl A with A on the edges: the face differences cancel in div B
        size = 0.3 * math.sqrt(2.0 / c["beta"]) * min(length) / (2 * math.pi)
        for comp in range(3):
            e1, e2 = (comp + 1) % 3, (comp + 2) % 3
            at = [np.append(lower[a], lower[a][-1] + d[a]) for a in range(3)]
            at[comp] = mid[comp]
            a = _waves(torch.zeros([len(v) for v in at[::-1]], device=dev), *at, length, rng, size)
            for axis, other, sign in ((e1, e2, -1.0), (e2, e1, 1.0)):  # dA/d(axis) goes to component `other`
                dim = 2 - axis
                w[5 + other].add_(torch.diff(a, dim=dim).narrow(2 - other, 0, shape[2 - other]), alpha=sign / d[axis])
    noise = torch.rand((3, shape[0], rows, shape[2]), device=dev, generator=gen)
    w[1:4, :, my:my + rows] += (2 * noise - 1) * (0.01 * cs)
    return w


class _Monitored(MHDSolver):
    """A program's solver: the diagnostics of the state before every step."""

    def monitor(self):
        self.log.append(self.diagnostics())
        return 0


def prepare(case, seed):
    if case["kind"] == "ensemble":
        boxes = _boxes(case, seed)
        configs = [_config(b) for b, _ in boxes]
        at = np.concatenate([[0], np.cumsum([8 * c.cells for c in configs])])
        # every state in one pinned host buffer, and one for the results
        first = torch.empty(int(at[-1]), pin_memory=True)
        last = torch.empty(int(at[-1]), pin_memory=True)
        for (b, s), i, j in zip(boxes, at, at[1:]):
            first[int(i):int(j)] = _state(b, s).reshape(-1).cpu()
        views = [[v.numpy()[i:j].reshape((8,) + c.shape) for c, i, j in zip(configs, at, at[1:])] for v in (first, last)]
        batch = BatchSolver(configs)
        batch.set_states(views[0])
        batch.autotune()
        batch.prepare(case["steps"])
        return dict(case=case, batch=batch, first=views[0], last=views[1], keep=(first, last))
    if case["kind"] == "slabs":
        n = case["slabs"]
        states = [_state(case, seed, r, n) for r in range(n)]
        group = SlabGroup(slab_config(_config(case), n), [s.cpu().numpy() for s in states])
        out = [torch.empty_like(s) for s in states]
        torch.cuda.synchronize()
        return dict(case=case, group=group, first=states, out=out)
    solver = (_Monitored if case["kind"] == "monitored" else MHDSolver)(_config(case))
    first = _state(case, seed)
    torch.cuda.synchronize()
    if case["kind"] == "adjoint":
        solver.set_state_device(first)
        solver.set_adjoint_tape_budget(case["budget"])
        grad = torch.empty(first.shape, pin_memory=True).numpy()
        return dict(case=case, solver=solver, grad=grad)
    solver.prepare(1 if case["kind"] == "monitored" else case["steps"])
    return dict(case=case, solver=solver, first=first, out=torch.empty_like(first))


def _window(case):
    return case["steps"] // 2 + 1, case["steps"]


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        state["batch"].set_states(state["first"])
        state["batch"].step(case["steps"])
        state["batch"].get_states(state["last"])
        boxes = state["last"]
        # the first boxes one by one, then all of them
        return {"boxes": [boxes[i] for i in range(min(8, len(boxes)))], "all": state["keep"][1]}
    if case["kind"] == "slabs":
        group = state["group"]
        for slab, first in zip(group.slabs, state["first"]):
            slab.set_state_device(first)
            slab.set_time(0.0, 0)
        group.step(case["steps"])
        for slab, out in zip(group.slabs, state["out"]):
            slab.get_state_device(out)
        return {"slabs": [dict(zip(FIELDS, out)) for out in state["out"]], "time": group.current_time()}
    solver = state["solver"]
    if case["kind"] == "adjoint":
        loss, grad, dt = solver.adjoint(case["steps"], window=_window(case), ckpt_every=case["ckpt"], out=state["grad"])
        return {"loss": loss, "gradient": dict(zip(FIELDS, grad)), "dt": dt}
    solver.set_state_device(state["first"])
    solver.set_time(0.0, 0)
    found = {}
    if case["kind"] == "monitored":
        solver.log = []
        solver.proceed(math.inf, max_steps=case["steps"])
        found["diagnostics"] = np.array([np.hstack([v for _, v in sorted(d.items())]) for d in solver.log])
    else:
        solver.step(case["steps"])
    solver.get_state_device(state["out"])
    return dict(zip(FIELDS, state["out"]), time=solver.current_time(), **found)


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how far results may be off


def _cells(case):
    if case["kind"] == "ensemble":
        return sum(_config(b).cells for b, _ in _boxes(case, 0))
    return case["nx"] * (case["ny"] + 2 * case["my"] * case.get("slabs", 1)) * (case["nz"] + 2 * case["mz"])


def work(case):
    """Per step and cell: the state read and written once (64 bytes); about 1150 float operations a stage (three faces
    of reconstruction, 110, and Riemann solver, 220; corner fields and face update, 60; conserved update, 100).
    The adjoint reverses what the forward does: twice its operations on top of it."""
    n = _cells(case) * case["steps"]
    stages = case.get("time_order", 2)
    if case["kind"] == "adjoint":
        return {"bytes": 64 * n, "flops": 3 * 1150 * stages * n}
    return {"bytes": 64 * n, "flops": 1150 * stages * n}


def tolerance(case):
    if case["kind"] == "adjoint":
        # against 64 bits: 6e-4 (listed) to 3e-3 (drawn), from the limiter, fan
        # and upwind choices that rounding moves
        return {"rel": 1e-3, "max": 0.3}
    if case.get("fast"):
        # against 64 bits: 6e-4, in the fields that start at zero
        return {"rel": 2e-3, "max": 0.3}
    if case["kind"] == "monitored":
        # the states are exact; the diagnostics are FP64 sums in any order
        return {"rel": 1e-12, "max": 1e-10}
    return "exact"  # every path of the step gives the reference's bits


# ---------------------------------------------------------------------------
# The scheme in 64 bits, in plain torch


def _at(a, axis, shift):
    """a at the index plus `shift` along x (0), y (1) or z (2), periodic."""
    return torch.roll(a, -shift, dims=a.dim() - 1 - axis)


def _faces(q, axis, order2):
    """Left and right states at the lower faces along `axis`."""
    b, c = _at(q, axis, -1), q
    if not order2:
        return b, c

    def smaller(u, v):
        return torch.where(u * v <= 0, torch.zeros_like(u), torch.where(u.abs() < v.abs(), u, v))
    d = q - _at(q, axis, -1)  # slope below each cell
    s = smaller(d, _at(d, axis, 1))  # limited slope of each cell
    return b + _at(s, axis, -1) / 2, c - s / 2


def _riemann(gamma, bn, left, right):
    """HLLD flux (mass, normal and transverse momenta, energy, transverse fields) from (rho, u, v, w, p, by, bz) pairs."""
    tiny = 1e-10
    sides = []
    for rho, u, v, w, p, by, bz in (left, right):
        b2 = bn * bn + by * by + bz * bz
        e = p / (gamma - 1) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * b2
        gp = gamma * p
        c = torch.sqrt((gp + b2 + torch.sqrt((gp + b2) ** 2 - 4 * gp * bn * bn)) / (2 * rho))
        sides.append(dict(rho=rho, u=u, v=v, w=w, p=p, by=by, bz=bz, e=e, c=c, pt=p + 0.5 * b2, vb=u * bn + v * by + w * bz))
    L, R = sides
    cmax = math.sqrt(2.0) * torch.maximum(L["c"], R["c"])
    L["s"] = torch.minimum(L["u"], R["u"]) - cmax
    R["s"] = torch.maximum(L["u"], R["u"]) + cmax
    L["d"], R["d"] = (L["s"] - L["u"]) * L["rho"], (R["s"] - R["u"]) * R["rho"]
    den = R["d"] - L["d"]
    sm = (R["d"] * R["u"] - L["d"] * L["u"] - R["pt"] + L["pt"]) / den
    pts = (R["d"] * L["pt"] - L["d"] * R["pt"] + L["d"] * R["d"] * (R["u"] - L["u"])) / den
    for S in sides:
        gap = S["s"] - sm
        S["rs"] = S["d"] / gap
        S["root"] = torch.sqrt(S["rs"])
        dn = S["d"] * gap - bn * bn + tiny
        turn, keep = bn * (sm - S["u"]) / dn, (S["rho"] * (S["s"] - S["u"]) ** 2 - bn * bn) / dn
        S["vs"], S["ws"] = S["v"] - S["by"] * turn, S["w"] - S["bz"] * turn
        S["bys"], S["bzs"] = S["by"] * keep, S["bz"] * keep
        S["vbs"] = sm * bn + S["vs"] * S["bys"] + S["ws"] * S["bzs"]
        S["es"] = ((S["s"] - S["u"]) * S["e"] - S["pt"] * S["u"] + pts * sm + bn * (S["vb"] - S["vbs"])) / gap
    L["alfven"], R["alfven"] = sm - bn.abs() / L["root"], sm + bn.abs() / R["root"]
    sign = torch.sign(bn)
    total, both = L["root"] + R["root"], L["root"] * R["root"]
    vss = (L["root"] * L["vs"] + R["root"] * R["vs"] + (R["bys"] - L["bys"]) * sign) / total
    wss = (L["root"] * L["ws"] + R["root"] * R["ws"] + (R["bzs"] - L["bzs"]) * sign) / total
    byss = (L["root"] * R["bys"] + R["root"] * L["bys"] + both * (R["vs"] - L["vs"]) * sign) / total
    bzss = (L["root"] * R["bzs"] + R["root"] * L["bzs"] + both * (R["ws"] - L["ws"]) * sign) / total
    vbss = sm * bn + vss * byss + wss * bzss
    zone = torch.full_like(sm, 5)
    for k, inside in ((4, (R["alfven"] <= 0) & (R["s"] >= 0)), (3, (sm <= 0) & (R["alfven"] >= 0)),
                      (2, (L["alfven"] <= 0) & (sm >= 0)), (1, (L["s"] <= 0) & (L["alfven"] >= 0)), (0, L["s"] > 0)):
        zone = torch.where(inside, torch.full_like(zone, k), zone)
    out = None
    for S, flip, mine in ((L, -1.0, (0, 1, 2)), (R, 1.0, (5, 4, 3))):
        rho, u, s, rs = S["rho"], S["u"], S["s"], S["rs"]
        ess = S["es"] + flip * S["root"] * (S["vbs"] - vbss) * sign
        plain = (rho * u, rho * u * u + S["pt"] - bn * bn, rho * S["v"] * u - bn * S["by"], rho * S["w"] * u - bn * S["bz"],
                 (S["e"] + S["pt"]) * u - bn * S["vb"], S["by"] * u - bn * S["v"], S["bz"] * u - bn * S["w"])
        own = (rho, rho * u, rho * S["v"], rho * S["w"], S["e"], S["by"], S["bz"])
        star = (rs, rs * sm, rs * S["vs"], rs * S["ws"], S["es"], S["bys"], S["bzs"])
        twin = (rs, rs * sm, rs * vss, rs * wss, ess, byss, bzss)
        fluxes = (plain, [f + s * (a - b) for f, a, b in zip(plain, star, own)],
                  [f + S["alfven"] * c - (S["alfven"] - s) * a - s * b for f, c, a, b in zip(plain, twin, star, own)])
        for k, values in zip(mine, fluxes):
            out = list(values) if out is None else [torch.where(zone == k, f, o) for f, o in zip(values, out)]
    return out


def _stage(geo, win, wb, dt):
    """One stage over `dt`: fluxes and corner fields from `win`, added to the conserved state of `wb`."""
    d, mid = (geo["dx"], geo["dy"], geo["dz"]), []
    ys = geo["corner_y"] + geo["dy"] * (torch.arange(win.shape[2], device=win.device, dtype=win.dtype) + 0.5)
    tide = (2 * geo["q"] * geo["omega"] ** 2 * ys)[None, :, None]
    for a in range(3):
        mid.append(0.5 * (win[5 + a] + _at(win[5 + a], a, 1)))
    pace, bflux = [0.0] * 5, {}
    for a in range(3):
        e1, e2 = (a + 1) % 3, (a + 2) % 3
        pairs = [_faces(q, a, geo["order2"]) for q in (win[0], win[1 + a], win[1 + e1], win[1 + e2], win[4], mid[e1], mid[e2])]
        left, right = [p[0] for p in pairs], [p[1] for p in pairs]
        if geo["shear"] and a < 2:
            other = win[2 - a]
            kick = 0.5 * (_at(other, a, -1) + other)
            kick = -2 * geo["omega"] * kick if a == 0 else 2 * geo["omega"] * kick + tide
            left[1], right[1] = left[1] + 0.5 * dt * kick, right[1] + 0.5 * dt * kick
        f = _riemann(geo["gamma"], win[5 + a], left, right)
        by_field = {0: f[0], 1 + a: f[1], 1 + e1: f[2], 1 + e2: f[3], 4: f[4]}
        for v in range(5):
            pace[v] = pace[v] + (by_field[v] - _at(by_field[v], a, 1)) / d[a]
        bflux[a, e1], bflux[a, e2] = f[5], f[6]

    def corner(a, b):
        """The flux of B_b along a on the edges of the a-b plane, upwind in v_b."""
        v, f1 = win[1 + b], bflux[a, b]
        wind = v + _at(v, b, -1)
        wind, f0 = wind + _at(wind, a, -1), _at(f1, b, -1)
        return torch.where(wind > 0, f0, torch.where(wind < 0, f1, 0.5 * (f0 + f1)))
    new = []
    for c in range(3):
        b = 0.0
        for o in range(3):
            if o != c:
                e = 0.5 * (corner(c, o) - corner(o, c))
                b = b + (_at(e, o, 1) - e) / d[o]
        new.append(wb[5 + c] + dt * b)

    def square(faces):
        return sum(b * b + _at(b, a, 1) ** 2 for a, b in enumerate(faces))
    gm1 = geo["gamma"] - 1
    rho = wb[0] + dt * pace[0]
    m = [wb[0] * wb[v] + dt * pace[v] for v in (1, 2, 3)]
    energy = wb[4] / gm1 + 0.5 * wb[0] * (wb[1] ** 2 + wb[2] ** 2 + wb[3] ** 2) + 0.25 * square(wb[5:8]) + dt * pace[4]
    p = (energy - 0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / rho - 0.25 * square(new)) * gm1
    vx, vy, vz = (v / rho for v in m)
    if geo["shear"]:
        vx, vy = vx - dt * 2 * geo["omega"] * vy, vy + dt * (2 * geo["omega"] * vx + tide)
    return torch.stack([rho, vx, vy, vz, p] + new)


def _fill(geo, ws, time):
    """The margins of every slab in `ws`: y rows from the neighbours, shifted by the shear, then z planes."""
    my, mz = geo["my"], geo["mz"]
    if my:
        shift = time * geo["rel_vel"]
        shift -= math.floor(shift / geo["extent_x"]) * geo["extent_x"]
        n = math.floor(shift / geo["dx"])
        up, down = [], []
        for w in ws:
            kick = torch.zeros((8, 1, 1, 1), dtype=w.dtype, device=w.device)
            kick[1] = geo["rel_vel"]
            up.append(torch.roll(w[:, :, -2 * my:-my], -n, dims=3) - kick)
            down.append(torch.roll(w[:, :, my:2 * my], n + 1, dims=3) + kick)
        filled = []
        for r, w in enumerate(ws):
            top = down[(r + 1) % len(ws)]
            edge = torch.cat([top[:6, :, :1], w[6:7, :, -my:w.shape[2] - my + 1], top[7:, :, :1]])
            filled.append(torch.cat([up[r - 1], w[:, :, my:-my], edge, top[:, :, 1:]], dim=2))
        ws = filled
    if mz:
        ws = [torch.cat([w[:, -2 * mz:-mz], w[:, mz:-mz], w[:, mz:2 * mz]], dim=1) for w in ws]
    return ws


def _time_step(geo, ws):
    least = math.inf
    for w in ws:
        b2 = sum(torch.maximum(w[5 + a] ** 2, _at(w[5 + a], a, 1) ** 2) for a in range(3))
        c = torch.sqrt((geo["gamma"] * w[4] + b2) / w[0])
        for a, h in enumerate((geo["dx"], geo["dy"], geo["dz"])):
            least = min(least, float((geo["cfl"] * h / (w[1 + a] + c).abs()).min()))
    return least


def _advance(geo, w, dt):
    if not geo["midpoint"]:
        return _stage(geo, w, w, dt)
    return _stage(geo, _stage(geo, w, w, dt / 2), w, dt)


def _integrate(geo, ws, steps, each=None):
    time = 0.0
    for _ in range(steps):
        if each is not None:
            each(ws[0])
        ws = _fill(geo, ws, time)
        dt = _time_step(geo, ws)
        ws = [_advance(geo, w, dt) for w in ws]
        time += dt
    return ws, time


def _inside(geo, w):
    return w[..., geo["mz"]:w.shape[-3] - geo["mz"], geo["my"]:w.shape[-2] - geo["my"], :]


def _stress(geo, w):
    return _inside(geo, -0.25 * (w[5] + _at(w[5], 0, 1)) * (w[6] + _at(w[6], 1, 1)))


def _diagnose(geo, w):
    """MHDSolver.diagnostics() as one row, by sorted name."""
    dv = geo["dx"] * geo["dy"] * geo["dz"]
    rho, vx, vy, vz, p = _inside(geo, w[:5])
    div = sum((_at(w[5 + a], a, 1) - w[5 + a]) / h for a, h in enumerate((geo["dx"], geo["dy"], geo["dz"])))
    mag = _inside(geo, 0.25 * sum(w[5 + a] ** 2 + _at(w[5 + a], a, 1) ** 2 for a in range(3))).sum() * dv
    kin, heat = (0.5 * rho * (vx ** 2 + vy ** 2 + vz ** 2)).sum() * dv, p.sum() * dv / (geo["gamma"] - 1)
    named = {"mass": rho.sum() * dv, "momentum": [(rho * v).sum() * dv for v in (vx, vy, vz)], "kinetic_energy": kin,
             "internal_energy": heat, "magnetic_energy": mag, "total_energy": kin + heat + mag, "bx2_mean": (w[5] ** 2).mean(),
             "by2_mean": (w[6] ** 2).mean(), "maxwell_stress": _stress(geo, w).mean(), "max_div_b": _inside(geo, div).abs().max(),
             "volume": rho.numel() * dv}
    return np.hstack([[float(x) for x in (v if isinstance(v, list) else [v])] for _, v in sorted(named.items())])


def exact(case, seed):
    if _cells(case) > 2.5e7:
        return None
    with torch.no_grad():
        if case["kind"] == "ensemble":
            found = []
            for c, s in _boxes(case, seed)[:8]:
                ws, _ = _integrate(_geometry(c), [_state(c, s).double()], c["steps"])
                found.append(ws[0].cpu())
            return {"boxes": found, "all": None}
        n = case.get("slabs", 1)
        geo = _geometry(case, n)
        ws = [_state(case, seed, r, n).double() for r in range(n)]
        if case["kind"] == "adjoint":
            return _exact_gradient(case, geo, ws[0])
        log = []
        ws, time = _integrate(geo, ws, case["steps"], (lambda w: log.append(_diagnose(geo, w))) if case["kind"] == "monitored" else None)
        if case["kind"] == "slabs":
            return {"slabs": [dict(zip(FIELDS, w)) for w in ws], "time": time}
        found = {"diagnostics": np.array(log)} if log else {}
        return dict(zip(FIELDS, ws[0]), time=time, **found)


def _exact_gradient(case, geo, w):
    first, last = _window(case)
    states, times, steps = [w], [0.0], []
    for _ in range(case["steps"]):
        w = _fill(geo, [states[-1]], times[-1])[0]
        steps.append(_time_step(geo, [w]))
        states.append(_advance(geo, w, steps[-1]))
        times.append(times[-1] + steps[-1])
    loss, grad = 0.0, torch.zeros_like(w)
    for n in range(case["steps"], -1, -1):
        with torch.enable_grad():
            x = states[n].clone().requires_grad_()
            value = _stress(geo, x).mean() / (last - first + 1)
            if first <= n <= last:
                loss += value.item()
                grad = grad + torch.autograd.grad(value, x)[0]
            if n > 0:
                x = states[n - 1].clone().requires_grad_()
                y = _advance(geo, _fill(geo, [x], times[n - 1])[0], steps[n - 1])
                grad = torch.autograd.grad(y, x, grad)[0]
    return {"loss": loss, "gradient": dict(zip(FIELDS, grad)), "dt": np.array(steps)}
