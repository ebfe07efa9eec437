"""The workloads this package is measured on, through its public entry points.

A case is a dict of plain values.  Its "kind" says which entry point it calls:

* ``step``      one ``SLChannelFlow.step_sl_bdf2`` (one channel, state on the GPU);
* ``advect``    one ``SLAdvector.advect`` (the drop-in advector called by itself);
* ``ensemble``  one ``ChannelEnsemble.step`` (several uneven channels together);
* ``gradient``  a rollout through ``SLRollout`` and its backward pass;
* ``host``      one ``HostStateStepper.step`` (state in pinned host memory).

The velocity fields follow the recipe of the package's own benchmark: the
Poiseuille profile plus the curl of a seeded random vector potential with
Fourier modes |k| <= 8 damped at the walls, scaled to a given rms (0.1 where
not said otherwise).  They are made on the GPU with plain torch.  Channels
that step are sent back to their initial state after SPAN steps (the
benchmark's default run), so that every pass works on a developed but
physical flow however many passes are taken.

``exact`` restates the step in plain float64 torch (dense z solves, searched
z intervals, torch.fft) without the package.
"""

import math

import torch
from torch.utils.checkpoint import checkpoint

from slchannel_b200 import SLAdvector, SLChannelFlow
from slchannel_b200.adjoint import SLRollout, kinetic_energy_loss
from slchannel_b200.ensemble import ChannelEnsemble
from slchannel_b200.host import HostStateStepper, pinned_like

DEFAULTS = {"Lx": 2 * math.pi, "Ly": math.pi, "Lz": 2.0, "gamma": 2.0, "Re": 2800.0, "urms": 0.1,
            "order": 6, "traj": 2, "precision": "fp64", "pressure": "noninc", "xy_rhs": "extrap",
            "stretching": "symmetric", "top": "dirichlet"}


SPAN = 20  # steps of one run of a channel before the next begins


def listed():
    big = {"kind": "step", "nx": 256, "ny": 256, "nz": 256, "Lx": 4 * math.pi, "Ly": 2 * math.pi,
           "Re": 2792.8, "dt": 0.01}
    return [
        # the smallest channels that are run in earnest: a first look at a flow,
        # a test, a parameter scan; latency and launches count
        {"name": "step_32_o4", "kind": "step", "nx": 32, "ny": 32, "nz": 32, "order": 4, "dt": 0.02},
        # the plain FP64 step of the package's first configuration
        {"name": "step_64_o6", "kind": "step", "nx": 64, "ny": 64, "nz": 64, "dt": 0.01},
        # an open channel on an odd grid: bottom-only stretching, free-slip top,
        # incremental pressure, about one cell per step
        {"name": "step_97x75x81_open_inc", "kind": "step", "nx": 97, "ny": 75, "nz": 81, "dt": 0.04,
         "stretching": "bottom", "top": "neumann", "pressure": "inc"},
        # the headline: the FP64 step at 256^3, triquintic, then tricubic
        dict(big, name="step_256_o6"),
        dict(big, name="step_256_o4", order=4),
        # the mixed-precision form of the same step, and its largest grid
        dict(big, name="step_256_mixed", precision="mixed", urms=0.12),
        dict(big, name="step_512x384x384_mixed", precision="mixed", nx=512, ny=384, nz=384, Re=5600.0,
             dt=0.005, urms=0.12),
        # the advector in someone else's solver: large steps (trajectory CFL 3)
        # and one more triple carried to the same feet
        {"name": "advect_128_cfl3_extra", "kind": "advect", "nx": 128, "ny": 128, "nz": 128,
         "dt": 0.1, "extra": 1},
        # an ensemble of uneven channels at trajectory CFL 3, in both forms
        # (a quarter of the benchmark's 48 channels)
        {"name": "ensemble_12_fp64", "kind": "ensemble", "n": 12, "draw": 4, "cfl": 3.0},
        {"name": "ensemble_12_mixed", "kind": "ensemble", "n": 12, "draw": 9, "cfl": 3.0,
         "precision": "mixed"},
        # the gradient of a rollout with recomputed segments (the benchmark's
        # grid and loss over fewer steps)
        {"name": "gradient_128x96x128", "kind": "gradient", "nx": 128, "ny": 96, "nz": 128, "dt": 0.01,
         "steps": 4, "every": 2},
        # the state lives in pinned host memory and crosses the bus every step
        {"name": "host_192x160x128", "kind": "host", "nx": 192, "ny": 160, "nz": 128, "dt": 0.01},
    ]


def _extent(rng, lo, hi):
    n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    # transforms like even sizes; a third of the grids keep whatever was drawn
    return n if rng.random() < 0.34 else max(lo, n - n % 8)


def draw(rng):
    """One more case of the same ranges: 16 to 384 cells per axis (up to 17 M
    points), trajectory CFL 0.1 to 3, every option the step has."""
    kind = rng.choices(["step", "advect", "ensemble", "gradient", "host"], [60, 10, 8, 12, 10])[0]
    if kind == "ensemble":
        return {"kind": "ensemble", "n": rng.randint(2, 12), "draw": rng.randrange(1 << 20),
                "cfl": round(math.exp(rng.uniform(math.log(0.3), math.log(3.0))), 3),
                "order": rng.choice([6, 6, 4]), "precision": rng.choice(["fp64", "mixed"])}
    most = {"step": 17e6, "advect": 4e6, "gradient": 1.2e6, "host": 8e6}[kind]
    size = math.exp(rng.uniform(math.log(8e3), math.log(most)))
    while True:
        nx, ny, nz = _extent(rng, 16, 384), _extent(rng, 16, 384), _extent(rng, 16, 384)
        if 0.8 * size <= nx * ny * nz <= min(1.25 * size, most):
            break
    cfl = math.exp(rng.uniform(math.log(0.1), math.log(3.0)))
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
            "dt": float("%.3g" % min(0.12, cfl * DEFAULTS["Lx"] / nx / 1.6)), "order": rng.choice([6, 6, 4]),
            "gamma": round(rng.uniform(1.6, 2.2), 3), "Re": round(rng.uniform(2000.0, 5600.0), 1)}
    if kind == "gradient":
        case["steps"] = rng.randint(1, 3)
        case["every"] = rng.randint(1, case["steps"])
        return case
    case["precision"] = rng.choice(["fp64", "fp64", "mixed"])
    case["traj"] = rng.choice([2, 2, 2, 4])
    if kind == "advect":
        case["extra"] = rng.randint(0, 2)
        return case
    if rng.random() < 0.3:
        case["stretching"] = "bottom"
    if rng.random() < 0.3:
        case["top"] = "neumann"
    if rng.random() < 0.2:
        case["xy_rhs"] = "lagged"
    if kind == "step" and rng.random() < 0.25:
        case["pressure"] = "inc"
    return case


def _full(case):
    return {**DEFAULTS, **{k: v for k, v in case.items() if k != "name"}}


def _members(case):
    """An ensemble's channels as step cases: sizes per axis from
    {32, 48, 64, 96, 128}, tanh gamma and Re uniform in their ranges."""
    g = torch.Generator().manual_seed(int(case["draw"]))

    def uni(lo, hi):
        return lo + (hi - lo) * float(torch.rand((), generator=g, dtype=torch.float64))

    out = []
    for i in range(int(case["n"])):
        nx, ny, nz = (int((32, 48, 64, 96, 128)[int(k)]) for k in torch.randint(0, 5, (3,), generator=g))
        out.append(_full({**case, "kind": "step", "nx": nx, "ny": ny, "nz": nz,
                          "gamma": uni(1.6, 2.2), "Re": uni(2000.0, 5000.0),
                          "dt": min(0.2, float(case["cfl"]) / max(1.7 * nx / DEFAULTS["Lx"], 0.35 * ny / DEFAULTS["Ly"])),
                          "member": i}))
    return out


# ----------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------
_F = {"dtype": torch.float64, "device": "cuda"}


def _z_grid(c):
    """Faces (nz+1) and centres with two ghosts (nz+2) of the tanh grid."""
    nz, g, Lz = c["nz"], c["gamma"], c["Lz"]
    s = torch.linspace(0.0, 1.0, nz + 1, dtype=torch.float64)
    if c["stretching"] == "bottom":
        zf = Lz * (1.0 - torch.tanh(g * (1.0 - s)) / math.tanh(g))
    else:
        zf = 0.5 * Lz * (1.0 + torch.tanh(g * (2.0 * s - 1.0)) / math.tanh(g))
    mid = 0.5 * (zf[:-1] + zf[1:])
    zc = torch.cat([-mid[:1], mid, (2.0 * zf[-1] - mid[-1]).reshape(1)])
    return zf.cuda(), zc.cuda()


def _velocity(c, seed, profile=True):
    """Interior (u, v, w): u and v (nx, ny, nz), w (nx, ny, nz-1)."""
    nx, ny, nz, Lz = c["nx"], c["ny"], c["nz"], c["Lz"]
    zf, zc = _z_grid(c)
    g = torch.Generator().manual_seed(int(seed) * 131 + int(c.get("member", 0)))
    K = 24  # modes that the grid resolves
    most = [min(8, e // 4) for e in (nx, ny, nz)]
    m = torch.stack([torch.randint(-k, k + 1, (3, K), generator=g) for k in most[:2]], 1).double()
    l = torch.randint(0, most[2] + 1, (3, K), generator=g).double()
    ph = 2 * math.pi * torch.rand((3, 2, K), generator=g, dtype=torch.float64)
    amp = torch.randn((3, K), generator=g, dtype=torch.float64) / (1 + (m.square().sum(1) + l.square()).sqrt())
    m, l, ph, amp = (t.cuda() for t in (m, l, ph, amp))

    def factor(k, phase, x, d):  # cos(k x + phase) or its derivative, (len(x), K)
        a = x[:, None] * k[None] + phase[None]
        return -k[None] * torch.sin(a) if d else torch.cos(a)

    def potential(a, x, y, z, der):
        kx, ky = 2 * math.pi * m[a, 0] / c["Lx"], 2 * math.pi * m[a, 1] / c["Ly"]
        kz = math.pi * l[a] / Lz
        D, dD = (z * (Lz - z)).square(), 2 * z * (Lz - z) * (Lz - 2 * z)
        Z = factor(kz, 0.0 * kz, z, False)
        Zz = (dD[:, None] * Z + D[:, None] * factor(kz, 0.0 * kz, z, True)) if der == 2 else D[:, None] * Z
        xy = (amp[a] * factor(kx, ph[a, 0], x, der == 0))[:, None, :] * factor(ky, ph[a, 1], y, der == 1)[None]
        return (xy.reshape(-1, xy.shape[-1]) @ Zz.T).reshape(len(x), len(y), len(z))

    dx, dy = c["Lx"] / nx, c["Ly"] / ny
    xf, yf = torch.arange(1, nx + 1, **_F) * dx, torch.arange(1, ny + 1, **_F) * dy
    xc, yc = xf - 0.5 * dx, yf - 0.5 * dy
    zi, zw = zc[1:-1], zf[1:-1]
    u = potential(2, xf, yc, zi, 1) - potential(1, xf, yc, zi, 2)
    v = potential(0, xc, yf, zi, 2) - potential(2, xc, yf, zi, 0)
    w = potential(1, xc, yc, zw, 0) - potential(0, xc, yc, zw, 1)
    rms = ((u.square().mean() + v.square().mean() + w.square().mean()) / 3).sqrt()
    u, v, w = (t * (c["urms"] / rms) for t in (u, v, w))
    if profile:
        u += 1.5 * (1.0 - (2.0 * zi / Lz - 1.0).square())
    return u, v, w


def _ghosted(c, u, v, w):
    """The package's ghost-shaped arrays of interior (u, v, w): periodic in x
    and y, no slip (or free slip at the top), no flow through the walls."""
    top = 1.0 if c["top"] == "neumann" else -1.0

    def walls(f):
        return torch.cat([-f[:, :, :1], f, top * f[:, :, -1:]], 2)

    def left(f, d):
        return torch.cat([f.narrow(d, f.shape[d] - 1, 1), f], d)

    def both(f, d):
        return torch.cat([f.narrow(d, f.shape[d] - 1, 1), f, f.narrow(d, 0, 1)], d)

    zero = torch.zeros_like(w[:, :, :1])
    return (left(both(walls(u), 1), 0).contiguous(), both(left(walls(v), 1), 0).contiguous(),
            both(both(torch.cat([zero, w, zero], 2), 1), 0).contiguous())


def _config(c):
    return {
        "grid": {"nx": c["nx"], "ny": c["ny"], "nz": c["nz"]},
        "domain": {"Lx": c["Lx"], "Ly": c["Ly"], "Lz": c["Lz"], "stretching_type": c["stretching"]},
        "flow": {"Re": c["Re"], "Re_tau": 180.0, "U_bulk": 1.0, "gamma": c["gamma"]},
        "boundary_conditions": {"top_wall": {"type": c["top"]}},
        "initialization": {"type": "parabolic"},
        "time": {"dt": c.get("dt", 0.01), "dt_update_interval": 0},
        "compute": {"device": "cuda"},
        "sl": {"interp_order": c["order"], "traj_interp_order": c["traj"], "n_traj_iters": 2,
               "interp_dtype": c["precision"], "bdf2_pressure": c["pressure"], "bdf2_xy_rhs": c["xy_rhs"]},
    }


def _flow(c, seed):
    """A channel with its initial field set and its BDF1 bootstrap step taken,
    and that initial field."""
    flow = SLChannelFlow(config=_config(c))
    V0 = _ghosted(c, *_velocity(c, seed))
    flow.set_state(*V0)
    flow.step_sl_bdf2(c["dt"])
    return flow, V0


def _mask(c, seed):
    """Smooth weights in (0, 1) at the interior positions."""
    f = dict(c, urms=1.0)
    return [torch.sigmoid(t) for t in _velocity(f, seed + 7, profile=False)]


def _advect_inputs(c, seed):
    triples = [_ghosted(c, *_velocity(c, seed * 17 + i)) for i in range(1 + int(c["extra"]))]
    mid = _ghosted(c, *_velocity(c, seed * 17 + 99))
    return triples, mid


def prepare(case, seed):
    c = _full(case)
    if c["kind"] == "step":
        flow, V0 = _flow(c, seed)
        return {"c": c, "flow": flow, "V0": V0, "done": 0}
    if c["kind"] == "advect":
        zf, zc = _z_grid(c)
        adv = SLAdvector(c["nx"], c["ny"], c["nz"], c["Lx"] / c["nx"], c["Ly"] / c["ny"], c["Lx"], c["Ly"],
                         c["Lz"], zf, zc, c["gamma"], stretching_type=c["stretching"], order=c["order"],
                         traj_order=c["traj"], n_traj_iters=2, top_wall_bc_type=c["top"],
                         interp_dtype=c["precision"], device="cuda")
        triples, mid = _advect_inputs(c, seed)
        return {"c": c, "adv": adv, "f": triples[0], "mid": mid, "extra": triples[1:]}
    if c["kind"] == "ensemble":
        members = _members(c)
        flows = [_flow(m, seed)[0] for m in members]
        ens = ChannelEnsemble(flows, [m["dt"] for m in members])
        first = [[t.clone() for t in (*ens.history(i), *ens.velocity(i))] for i in range(ens.n)]
        return {"c": c, "ens": ens, "first": first, "done": 0}
    if c["kind"] == "gradient":
        flow = SLChannelFlow(config=_config(c))
        return {"c": c, "flow": flow, "V0": _ghosted(c, *_velocity(c, seed)), "mask": _mask(c, seed)}
    flow, _ = _flow(c, seed)
    first = [[pinned_like(t).copy_(t) for t in level]
             for level in ((flow.u_nm1, flow.v_nm1, flow.w_nm1), (flow.u, flow.v, flow.w))]
    ring = [[pinned_like(t).zero_() for t in first[0]] for _ in range(3)]
    return {"c": c, "stepper": HostStateStepper(flow), "first": first, "ring": ring, "done": 0,
            "p": pinned_like(flow.p).copy_(flow.p), "bulk": torch.zeros(2, dtype=torch.float64).pin_memory()}


def _bulk(c, both):
    """[u_bulk, forcing] pairs.  The forcing is the bulk velocity's tiny
    defect over dt: in the mixed form it is the sum of the FP32 rounding of a
    step, which has no value to compare, so only the bulk velocity is given."""
    return both if c["precision"] == "fp64" else both.view(-1, 2)[:, 0]


def run(state):
    c = state["c"]
    if c["kind"] == "step":
        flow = state["flow"]
        if state["done"] == SPAN:
            flow.set_state(*state["V0"])
            flow.step_sl_bdf2(c["dt"])
            state["done"] = 0
        state["done"] += 1
        bulk, forcing = flow.step_sl_bdf2(c["dt"])
        return {"V": (flow.u, flow.v, flow.w), "p": flow.p,
                "bulk": (bulk, forcing) if c["precision"] == "fp64" else bulk}
    if c["kind"] == "advect":
        adv, extra = state["adv"], state["extra"]
        out = adv.advect(*state["f"], *state["mid"], c["dt"], extra_rhs=extra if extra else None)
        return {"out": out[:3], "extra": out[3] if extra else []}
    if c["kind"] == "ensemble":
        ens = state["ens"]
        if state["done"] == SPAN:
            for i, first in enumerate(state["first"]):
                for t, t0 in zip((*ens.history(i), *ens.velocity(i)), first):
                    t.copy_(t0)
            state["done"] = 0
        state["done"] += 1
        ens.step()
        return {"V": [ens.velocity(i) for i in range(ens.n)], "p": ens.p, "bulk": _bulk(c, ens.bulk_out)}
    if c["kind"] == "gradient":
        V0 = [t.detach().requires_grad_(True) for t in state["V0"]]
        VN = SLRollout.apply(*V0, state["flow"], c["dt"], c["steps"], c["every"])
        J = kinetic_energy_loss(VN, state["mask"], state["flow"])
        grads = torch.autograd.grad(J, V0)
        return {"J": J.detach(), "V": [t.detach() for t in VN], "grad": grads}
    k = state["done"] % SPAN
    state["done"] += 1
    level = lambda i: state["first"][i + 2] if i < 0 else state["ring"][i % 3]  # noqa: E731
    prev, cur, nxt = level(k - 2), level(k - 1), level(k)
    state["stepper"].step(cur, prev, nxt, state["p"], state["bulk"], c["dt"])
    return {"V": nxt, "p": state["p"], "bulk": _bulk(c, state["bulk"])}


def work(case):
    c = _full(case)
    if c["kind"] == "ensemble":
        parts = [work(m) for m in _members(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = c["nx"] * c["ny"] * c["nz"]
    O, T = c["order"], c["traj"]
    # per foot: the separable contraction and its weights; per trajectory
    # sample: three such contractions of the trajectory order
    foot = 2 * (O**3 + O**2 + O) + 12 * O
    sample = 3 * (2 * (T**3 + T**2 + T) + 6 * T)
    trace = sample + 20
    fft = 2 * 2.5 * math.log2(c["nx"] * c["ny"])
    step = 3 * (2 * (foot + trace) + sample + 30) + 3 * 10 + fft + 60
    if c["kind"] == "advect":
        k = 1 + c["extra"]
        return {"bytes": 8.0 * n * 3 * (2 * k + 1), "flops": float(n) * 3 * (k * foot + trace + sample)}
    if c["kind"] == "gradient":
        # every step forward; every step backward: its state and adjoint read,
        # two adjoints updated, about three times the forward's arithmetic
        return {"bytes": 8.0 * n * c["steps"] * (9 + 15), "flops": float(n) * c["steps"] * 4 * step}
    # V^n and V^{n-1} read, V^{n+1} and p written (inc: two pressures read, too)
    return {"bytes": 8.0 * n * (10 + (2 if c["pressure"] == "inc" else 0)), "flops": float(n) * step}


# ----------------------------------------------------------------------
# The same in plain float64 torch
# ----------------------------------------------------------------------
class _Plain:
    """The SL-BDF2 step on interior (u, v, w), differentiable."""

    CHUNK = 6_000_000

    def __init__(self, c):
        self.c = c
        self.n = (c["nx"], c["ny"], c["nz"])
        self.zf, self.zc = _z_grid(c)
        self.dzf, self.dzc = self.zf.diff(), self.zc.diff()
        self.dx, self.dy = c["Lx"] / c["nx"], c["Ly"] / c["ny"]
        self.nu, self.top = 1.0 / c["Re"], 1.0 if c["top"] == "neumann" else -1.0
        self.lo = float(self.zf[0]) + 1e-12 * c["Lz"]
        self.hi = float(self.zf[-1]) - 1e-12 * c["Lz"]
        self.shift = ((0.0, -0.5), (-0.5, 0.0), (-0.5, -0.5))

    def nodes(self, V):
        """The three components on their node grids (x, y periodic)."""
        u, v, w = V
        walls = lambda f: torch.cat([-f[:, :, :1], f, self.top * f[:, :, -1:]], 2)  # noqa: E731
        zero = torch.zeros_like(w[:, :, :1])
        return (walls(u).roll(1, 0).contiguous(), walls(v).roll(1, 1).contiguous(),
                torch.cat([zero, w, zero], 2).contiguous())

    @staticmethod
    def _lagrange(x, nodes):
        out = []
        for m in range(len(nodes)):
            f = torch.ones_like(x)
            for k in range(len(nodes)):
                if k != m:
                    f = f * ((x - nodes[k]) / (nodes[m] - nodes[k]))
            out.append(f)
        return out

    def interp(self, F, comp, order, x, y, z):
        nx, ny, _ = self.n
        zn = self.zf if comp == 2 else self.zc
        h = order // 2 - 1
        offs = [float(m - h) for m in range(order)]
        s = x / self.dx + self.shift[comp][0]
        bx = s.detach().floor()
        wx = self._lagrange(s - bx, offs)
        s = y / self.dy + self.shift[comp][1]
        by = s.detach().floor()
        wy = self._lagrange(s - by, offs)
        # faces locate the cell; centres then choose between two of its intervals
        zd = z.detach().contiguous()
        cell = (torch.searchsorted(self.zf, zd, right=True) - 1).clamp(0, self.n[2] - 1)
        m0 = cell if comp == 2 else cell + (zd >= self.zc[cell + 1]).long()
        k0 = (m0 - h).clamp(0, len(zn) - order)
        wz = self._lagrange(z, [zn[k0 + m] for m in range(order)])
        ix = [((bx.long() + (m - h)) % nx) * F.stride(0) for m in range(order)]
        iy = [((by.long() + (m - h)) % ny) * F.stride(1) + k0 for m in range(order)]
        flat, acc = F.reshape(-1), 0.0
        for i in range(order):
            a = 0.0
            for j in range(order):
                at = ix[i] + iy[j]
                b = 0.0
                for k in range(order):
                    b = b + wz[k] * flat[at + k]
                a = a + wy[j] * b
            acc = acc + wx[i] * a
        return acc

    def feet(self, M, comp, i0, i1, depths):
        ny = self.n[1]
        sx, sy = self.shift[comp]
        x = ((torch.arange(i0, i1, **_F) + (1.0 + sx)) * self.dx).view(-1, 1, 1)
        y = ((torch.arange(ny, **_F) + (1.0 + sy)) * self.dy).view(1, -1, 1)
        z = (self.zf[1:-1] if comp == 2 else self.zc[1:-1]).view(1, 1, -1)
        x, y, z = (t.reshape(-1) for t in torch.broadcast_tensors(x, y, z))
        T = self.c["traj"]
        first = [self.interp(M[q], q, T, x, y, z.clamp(self.lo, self.hi)) for q in range(3)]
        out = []
        for dt in depths:
            v = first
            for it in range(2):
                xm, ym = x - 0.5 * dt * v[0], y - 0.5 * dt * v[1]
                zm = (z - 0.5 * dt * v[2]).clamp(self.lo, self.hi)
                if it == 0:
                    v = [self.interp(M[q], q, T, xm, ym, zm) for q in range(3)]
            out.append((2 * xm - x, 2 * ym - y, (2 * zm - z).clamp(self.lo, self.hi)))
        return out

    def along(self, fields, M, depths, grad=False):
        """Field f of `fields` (node triples) at the feet of depth depths[f]
        (or all at the one depth given)."""
        nx, ny, nz = self.n
        out = [[] for _ in fields]
        for comp in range(3):
            per = ny * (nz - 1 if comp == 2 else nz)
            step = max(1, self.CHUNK // per)
            got = [[] for _ in fields]
            for i0 in range(0, nx, step):
                i1 = min(nx, i0 + step)

                def part(*a, i0=i0, i1=i1, comp=comp):
                    Fs, Ms = a[:len(fields)], a[len(fields):]
                    feet = self.feet(Ms, comp, i0, i1, depths)
                    return tuple(self.interp(f, comp, self.c["order"], *feet[min(k, len(feet) - 1)])
                                 for k, f in enumerate(Fs))

                args = [f[comp] for f in fields] + list(M)
                res = checkpoint(part, *args, use_reentrant=False) if grad else part(*args)
                for k, r in enumerate(res):
                    got[k].append(r.reshape(i1 - i0, ny, -1))
            for k in range(len(fields)):
                out[k].append(torch.cat(got[k]))
        return out

    def diffuse(self, f):
        return self.nu * ((f.roll(-1, 0) - 2 * f + f.roll(1, 0)) / self.dx**2
                          + (f.roll(-1, 1) - 2 * f + f.roll(1, 1)) / self.dy**2)

    def zsolve(self, f, comp, dt):
        nz, a = self.n[2], dt * self.nu
        if comp == 2:
            dl, dr, dc = self.dzf[:-1], self.dzf[1:], self.dzc[1:-1]
        else:
            dl, dr, dc = self.dzc[:-1], self.dzc[1:], self.dzf
        low, up = -a / (dl * dc), -a / (dr * dc)
        mid = 1.0 - low - up
        if comp != 2:
            mid = mid.clone()
            mid[0] -= low[0]
            mid[-1] += self.top * up[-1]
        A = torch.diag(mid) + torch.diag(low[1:], -1) + torch.diag(up[:-1], 1)
        n = f.shape
        return torch.linalg.solve(A, f.reshape(-1, n[2]).T).T.reshape(n).contiguous()

    def poisson(self, rhs):
        nx, ny, nz = self.n
        kx = torch.fft.fftfreq(nx, 1.0 / nx, **_F) * (math.pi / nx)
        ky = torch.arange(ny // 2 + 1, **_F) * (math.pi / ny)
        k2 = ((2 / self.dx * kx.sin()).square()[:, None] + (2 / self.dy * ky.sin()).square()[None]).reshape(-1)
        left, right = 1.0 / (self.dzc[:-1] * self.dzf), 1.0 / (self.dzc[1:] * self.dzf)
        h = torch.fft.rfft2(rhs, dim=(0, 1))
        shape = h.shape
        h = h.reshape(-1, nz)
        cp, dp = [], []
        for k in range(nz):
            b = -(left[k] + right[k] + k2)
            b = b + left[k] if k == 0 else b
            b = b + right[k] if k == nz - 1 else b
            sup = (right[k] if k < nz - 1 else right[k] * 0) * torch.ones_like(k2)
            if k == 0:  # the mean mode's first row is the identity
                b, sup = torch.cat([torch.ones_like(b[:1]), b[1:]]), torch.cat([sup[:1] * 0, sup[1:]])
                cp.append(sup / b)
                dp.append(h[:, k] / b)
            else:
                d = b - left[k] * cp[-1]
                dp.append((h[:, k] - left[k] * dp[-1]) / d)
                cp.append(sup / d)
        x = [dp[-1]]
        for k in range(nz - 2, -1, -1):
            x.append(dp[k] - cp[k] * x[-1])
        return torch.fft.irfft2(torch.stack(x[::-1], 1).reshape(shape), s=(nx, ny), dim=(0, 1))

    def minus_grad(self, V, phi, dt):
        u, v, w = V
        return (u - dt * (phi.roll(-1, 0) - phi) / self.dx, v - dt * (phi.roll(-1, 1) - phi) / self.dy,
                w - dt * phi.diff(dim=2) / self.dzc[1:-1])

    def finish(self, V, dt, p_ext=None):
        """The predictor V to the next velocity: z diffusion, projection,
        bulk shift.  Returns (V, phi, forcing * step)."""
        if p_ext is not None:
            V = self.minus_grad(V, p_ext, dt)
        u, v, w = (self.zsolve(f, q, dt) for q, f in enumerate(V))
        zero = torch.zeros_like(w[:, :, :1])
        div = ((u - u.roll(1, 0)) / self.dx + (v - v.roll(1, 1)) / self.dy
               + torch.cat([zero, w, zero], 2).diff(dim=2) / self.dzf)
        phi = self.poisson(div / dt)
        u, v, w = self.minus_grad((u, v, w), phi, dt)
        vol = self.dx * self.dy * self.dzf / (self.c["Lx"] * self.c["Ly"] * self.c["Lz"])
        shift = 1.0 - (u.sum((0, 1)) * vol).sum()
        return (u + shift, v, w), phi, shift

    def bdf1(self, V, dt, grad=False):
        N = self.nodes(V)
        (adv,) = self.along([N], N, [dt], grad)
        return self.finish([a + dt * self.diffuse(f) for a, f in zip(adv, V)], dt)

    def bdf2(self, V, W, dt, p_ext=None, grad=False):
        star = [2 * a - b for a, b in zip(V, W)]
        near, far = self.along([self.nodes(V), self.nodes(W)], self.nodes(star), [dt, 2 * dt], grad)
        R = [self.diffuse(f) for f in (V if self.c["xy_rhs"] == "lagged" else star)]
        e = 2.0 / 3.0 * dt
        return self.finish([4.0 / 3.0 * a - b / 3.0 + e * r for a, b, r in zip(near, far, R)], e, p_ext)

    def pressure(self, phi):
        f = torch.cat([phi[:, :, :1], phi, phi[:, :, -1:]], 2)
        f = torch.cat([f[:, -1:], f, f[:, :1]], 1)
        return torch.cat([f[-1:], f, f[:1]], 0)

    def two_steps(self, seed):
        """(ghost-shaped V^2, p, [u_bulk, forcing]) of the channel _flow makes."""
        c, dt = self.c, self.c["dt"]
        V0 = _velocity(c, seed)
        V1, p1, _ = self.bdf1(V0, dt)
        inc = c["pressure"] == "inc"
        V2, phi, shift = self.bdf2(V1, V0, dt, p1 if inc else None)
        p = self.pressure(phi) + (self.pressure(p1) if inc else 0.0)
        return _ghosted(c, *V2), p, torch.stack([torch.ones_like(shift), shift / dt])


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "ensemble":
        got = [_Plain(m).two_steps(seed) for m in _members(c)]
        return {"V": [g[0] for g in got], "p": [g[1] for g in got],
                "bulk": _bulk(c, torch.cat([g[2] for g in got]))}
    plain = _Plain(c)
    if c["kind"] == "step":
        V, p, b = plain.two_steps(seed)
        return {"V": V, "p": p, "bulk": (b[0], b[1]) if c["precision"] == "fp64" else b[0]}
    if c["kind"] == "host":
        V, p, b = plain.two_steps(seed)
        return {"V": V, "p": p, "bulk": _bulk(c, b)}
    if c["kind"] == "advect":
        # what lies outside the interiors of the advector's buffers is not refreshed
        triples, mid = _advect_inputs(c, seed)
        cut = lambda t: (t[0][1:, 1:-1, 1:-1], t[1][1:-1, 1:, 1:-1], t[2][1:-1, 1:-1, 1:-1])  # noqa: E731
        M = plain.nodes(cut(mid))
        got = plain.along([plain.nodes(cut(t)) for t in triples], M, [c["dt"]])
        pad = torch.nn.functional.pad
        out = (pad(got[0][0], (1, 1, 1, 1, 1, 0)), pad(got[0][1], (1, 1, 1, 0, 1, 1)),
               pad(got[0][2], (1, 1, 1, 1, 1, 1)))
        return {"out": out, "extra": got[1:]}
    if c["nx"] * c["ny"] * c["nz"] * c["steps"] > 7_000_000:
        return None  # the recomputed graph of more steps takes too long
    ghosts = [t.requires_grad_(True) for t in _ghosted(c, *_velocity(c, seed))]
    mask = _mask(c, seed)
    V = (ghosts[0][1:, 1:-1, 1:-1], ghosts[1][1:-1, 1:, 1:-1], ghosts[2][1:-1, 1:-1, 1:-1])
    old, new = V, plain.bdf1(V, c["dt"], grad=True)[0]
    for _ in range(c["steps"] - 1):
        old, new = new, plain.bdf2(new, old, c["dt"], grad=True)[0]
    J = sum(0.5 * (m * f.square()).sum() for m, f in zip(mask, new))
    grads = torch.autograd.grad(J, ghosts)
    return {"J": J.detach(), "V": [t.detach() for t in _ghosted(c, *new)], "grad": grads}
