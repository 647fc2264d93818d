"""What is timed of this framework: the work that its users have it do, through its public entry
points, from the smallest grid that a run is made on to the headline one.

A case is a dict of plain values; its "kind" says which entry points it goes through:

* ``run``     a device-resident simulation advanced by the driver loop (``Context.run``), the state
              handed in and taken out as device planes;
* ``driver``  the reference driver's own loop: the CFL step read on the host, then one step, repeated
              (``Context.cfl_dt`` + ``Context.step``);
* ``host``    one step of a program that keeps its state in (pinned) host memory;
* ``rate``    the implicit resistive rate of a face field (``Context.resistive_rate``);
* ``batch``   many independent simulations of uneven sizes stepped together (``Batch.run``);
* ``grad``    forward and backward pass of a differentiable trajectory (``autograd.trajectory``).

Everything is FP64: the framework has no other type. Inputs are smooth periodic fields of random
phases and amplitudes (Orszag-Tang vortices for the single runs, sums of Fourier modes for the
ensembles and the gradients), made on the GPU from the seed alone.
"""
import math

import torch
import torch.utils.checkpoint

import magnetohydrodynamics_simulator_b200 as mhd
from magnetohydrodynamics_simulator_b200 import autograd as mhd_autograd

DEV = "cuda" if torch.cuda.is_available() else "cpu"
GAMMA = 5.0 / 3.0
COURANT, SAFETY = 0.4, 0.9
ARS_G = (2.0 - math.sqrt(2.0)) / 2.0
ARS_D = 1.0 - 1.0 / (2.0 * ARS_G)


def listed():
    return [
        # a student-size run stepped by the reference driver's own loop: launches and host waits
        {"name": "driver_64", "kind": "driver", "nx": 64, "ny": 64, "eta": 1e-3, "steps": 10},
        # the configured 128^2 Orszag-Tang run
        {"name": "run_128", "kind": "run", "nx": 128, "ny": 128, "eta": 1e-3, "steps": 20},
        # an ordinary production grid
        {"name": "run_512", "kind": "run", "nx": 512, "ny": 512, "eta": 1e-3, "steps": 10},
        # ragged sizes, dx != dy, a resistive plasma and the literal corner test
        {"name": "run_1000x700", "kind": "run", "nx": 1000, "ny": 700, "eta": 1e-2, "steps": 6,
         "aspect": 1.25, "true_abs": True},
        # the headline: 4096^2, eta 1e-4
        {"name": "run_4096", "kind": "run", "nx": 4096, "ny": 4096, "eta": 1e-4, "steps": 3},
        # the strongly resistive configuration (eta 10, fixed dt): the solves take most of the step
        {"name": "stiff_512", "kind": "run", "nx": 512, "ny": 512, "eta": 10.0, "steps": 2, "dt": 1e-3},
        # one implicit solve and its rate on a caller's device planes
        {"name": "rate_1024", "kind": "rate", "nx": 1024, "ny": 1024, "eta": 5e-3, "alpha_h2": 0.05},
        # an ensemble of small uneven runs, default decomposition
        {"name": "batch_small", "kind": "batch", "count": 24, "lo": 48, "hi": 160, "steps": 4, "tune": False},
        # the configured ensemble: 64 runs of 256^2 .. 1024^2, autotuned
        {"name": "batch_mixed", "kind": "batch", "count": 64, "lo": 256, "hi": 1024, "steps": 3, "tune": True},
        # gradients: a small inverse problem and the configured size
        {"name": "grad_256", "kind": "grad", "nx": 256, "ny": 256, "eta": 5e-3, "dt": 2e-3, "steps": 20, "every": 5},
        {"name": "grad_1024", "kind": "grad", "nx": 1024, "ny": 1024, "eta": 5e-3, "dt": 1e-3, "steps": 20, "every": 10},
        # a host program that moves its state over PCIe every step
        {"name": "host_1024", "kind": "host", "nx": 1024, "ny": 1024, "eta": 1e-3, "steps": 1},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "driver", "rate", "batch", "grad", "host", "stiff"])
    if kind == "run":
        nx, ny = int(_log(rng, 40, 2600)), int(_log(rng, 40, 2600))
        c = {"kind": "run", "nx": nx, "ny": ny, "eta": round(_log(rng, 1e-4, 1e-2), 6), "steps": rng.randint(2, 8)}
        if rng.random() < 0.5:
            c["aspect"] = round(rng.uniform(0.6, 1.6), 3)
        if rng.random() < 0.25:
            c["true_abs"] = True
        return c
    if kind == "stiff":
        n = int(_log(rng, 64, 700))
        return {"kind": "run", "nx": n, "ny": int(_log(rng, 64, 700)), "eta": round(_log(rng, 0.1, 10.0), 5),
                "steps": rng.randint(1, 3), "dt": 1e-3}
    if kind == "driver":
        return {"kind": "driver", "nx": int(_log(rng, 32, 400)), "ny": int(_log(rng, 32, 400)),
                "eta": round(_log(rng, 1e-4, 1e-2), 6), "steps": rng.randint(4, 12)}
    if kind == "rate":
        return {"kind": "rate", "nx": int(_log(rng, 40, 3000)), "ny": int(_log(rng, 40, 3000)),
                "eta": round(_log(rng, 1e-4, 1e-1), 6), "alpha_h2": round(_log(rng, 1e-3, 2.0), 5)}
    if kind == "batch":
        lo = int(_log(rng, 32, 300))
        return {"kind": "batch", "count": rng.randint(4, 80), "lo": lo, "hi": int(lo * rng.uniform(1.2, 3.0)),
                "steps": rng.randint(2, 5), "tune": rng.random() < 0.5}
    if kind == "grad":
        return {"kind": "grad", "nx": int(_log(rng, 64, 900)), "ny": int(_log(rng, 64, 900)),
                "eta": round(_log(rng, 1e-3, 1e-2), 6), "dt": 1e-3, "steps": rng.randint(6, 16),
                "every": rng.randint(2, 6)}
    return {"kind": "host", "nx": int(_log(rng, 200, 2000)), "ny": int(_log(rng, 200, 2000)),
            "eta": round(_log(rng, 1e-4, 1e-2), 6), "steps": 1}


# ------------------------------------------------------------------------------------- inputs


def _spacing(case):
    """Periodic box of 2 pi (x) by 2 pi * aspect (y)."""
    return 2 * math.pi / case["nx"], 2 * math.pi * case.get("aspect", 1.0) / case["ny"]


def _gen(seed):
    return torch.Generator(device="cpu").manual_seed(int(seed))


def _phases(g, n):
    return (2 * math.pi * torch.rand(n, generator=g, dtype=torch.float64)).tolist()


def _modes(g, nx, ny, count, lo, hi, kmax, shift):
    """Sum of `count` Fourier modes |k| <= kmax with amplitudes in [lo, hi], sampled at index + shift."""
    x = (2 * math.pi / nx) * (torch.arange(nx, device=DEV, dtype=torch.float64) + shift)
    y = (2 * math.pi / ny) * (torch.arange(ny, device=DEV, dtype=torch.float64) + shift)
    f = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
    for _ in range(count):
        kx, ky = 0, 0
        while kx == 0 and ky == 0:
            kx, ky = torch.randint(-kmax, kmax + 1, (2,), generator=g).tolist()
        amp, ph = torch.rand(2, generator=g, dtype=torch.float64).tolist()
        amp, ph = lo + (hi - lo) * amp, 2 * math.pi * ph
        a, b = kx * x + ph, ky * y
        f += amp * (torch.sin(a)[None, :] * torch.cos(b)[:, None] + torch.cos(a)[None, :] * torch.sin(b)[:, None])
    return f


def _state(rho, vx, vy, p, az, dx, dy):
    """Conserved planes (6, ny, nx); face B is the discrete curl of the corner potential az."""
    bx = (torch.roll(az, -1, 0) - az) / dy
    by = -(torch.roll(az, -1, 1) - az) / dx
    bxc = 0.5 * (bx + torch.roll(bx, -1, 1))
    byc = 0.5 * (by + torch.roll(by, -1, 0))
    E = p / (GAMMA - 1.0) + 0.5 * rho * (vx * vx + vy * vy) + 0.5 * (bxc * bxc + byc * byc)
    return torch.stack([rho, rho * vx, rho * vy, E, bx, by])


def _vortex(nx, ny, dx, dy, seed):
    """An Orszag-Tang vortex with random phases and a few per cent of smooth density and pressure modes."""
    g = _gen(seed)
    ph = _phases(g, 4)
    x = (2 * math.pi / nx) * torch.arange(nx, device=DEV, dtype=torch.float64)
    y = (2 * math.pi / ny) * torch.arange(ny, device=DEV, dtype=torch.float64)
    az = 0.5 * torch.cos(2 * x + ph[0])[None, :] + torch.cos(y + ph[1])[:, None]
    vx = -torch.sin(y + math.pi / ny + ph[2])[:, None] + _modes(g, nx, ny, 2, 0.02, 0.1, 4, 0.5)
    vy = torch.sin(x + math.pi / nx + ph[3])[None, :] + _modes(g, nx, ny, 2, 0.02, 0.1, 4, 0.5)
    rho = (25.0 / 9.0) * (1.0 + _modes(g, nx, ny, 3, 0.01, 0.04, 6, 0.5))
    p = (5.0 / 3.0) * (1.0 + _modes(g, nx, ny, 3, 0.01, 0.04, 6, 0.5))
    return _state(rho, vx, vy, p, az, dx, dy)


def _member(nx, ny, dx, dy, seed):
    """One ensemble member: smooth random density, velocity and potential of 8 modes each."""
    g = _gen(seed)
    rho = torch.clamp(1.0 + _modes(g, nx, ny, 6, 0.02, 0.12, 8, 0.5), min=0.2)
    vx = _modes(g, nx, ny, 8, 0.1, 1.0, 3, 0.5)
    vy = _modes(g, nx, ny, 8, 0.1, 1.0, 3, 0.5)
    az = _modes(g, nx, ny, 8, 0.1, 1.0, 3, 0.0)
    p = 1.0 + _modes(g, nx, ny, 3, 0.01, 0.05, 4, 0.5)
    return _state(rho, vx, vy, p, az, dx, dy)


def _smooth(nx, ny, dx, dy, seed):
    """The gradient's state: 4 modes of velocity 0.05 and potential 0.1 on a nearly uniform gas."""
    g = _gen(seed)
    vx = _modes(g, nx, ny, 4, 0.025, 0.05, 4, 0.5)
    vy = _modes(g, nx, ny, 4, 0.025, 0.05, 4, 0.5)
    az = _modes(g, nx, ny, 4, 0.05, 0.1, 4, 0.0)
    rho = 1.0 + _modes(g, nx, ny, 3, 0.01, 0.03, 4, 0.5)
    p = 1.0 + _modes(g, nx, ny, 3, 0.01, 0.03, 4, 0.5)
    u0 = _state(rho, vx, vy, p, az, dx, dy)
    # the observed state that the misfit is taken against: the same gas with other modes
    target = _state(rho, 0.9 * vx, 0.9 * vy, p, az + _modes(g, nx, ny, 2, 0.005, 0.01, 4, 0.0), dx, dy)
    return u0, target


def _ptrs(t):
    return [t[k].data_ptr() for k in range(t.shape[0])]


def _ensemble(case, seed):
    """(n, eta, seed) of every member: sizes in steps of the box [lo, hi], eta log-uniform in [1e-4, 1e-2].
    The sizes depend on the case alone: an ensemble's decomposition does not change with its data."""
    g = _gen(1000003 * case["count"] + 1009 * case["lo"] + case["hi"])
    out = []
    for k in range(case["count"]):
        u, v = torch.rand(2, generator=g, dtype=torch.float64).tolist()
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** u))
        n += n % 2 if k % 3 else 0  # most grids are even, some odd
        n = max(case["lo"], min(case["hi"], n))
        out.append((n, math.exp(math.log(1e-4) + v * math.log(100.0)), 7919 * int(seed) + k))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        members = _ensemble(case, seed)
        s["u0"] = [_member(n, n, 2 * math.pi / n, 2 * math.pi / n, sd) for n, _, sd in members]
        # one buffer for all members' final planes, and each member's part of it
        s["all"] = torch.empty(sum(u.numel() for u in s["u0"]), device=DEV, dtype=torch.float64)
        s["out"] = [o.view_as(u) for o, u in zip(s["all"].split([u.numel() for u in s["u0"]]), s["u0"])]
        b = mhd.Batch([{"nx": n, "ny": n, "dx": 2 * math.pi / n, "dy": 2 * math.pi / n, "eta": eta,
                        "courant": COURANT, "safety": SAFETY} for n, eta, _ in members])
        torch.cuda.synchronize()
        s["batch"] = b
        if case["tune"]:
            for i, u in enumerate(s["u0"]):
                b.set_state_device(i, _ptrs(u))
            b.autotune()
        return s
    nx, ny = case["nx"], case["ny"]
    dx, dy = _spacing(case)
    if kind == "grad":
        s["u0"], s["target"] = _smooth(nx, ny, dx, dy, seed)
        s["eta"] = torch.tensor(case["eta"], dtype=torch.float64)
        s["adj"] = mhd.Adjoint(nx, ny, dx, dy, case["eta"], case["dt"], case["steps"], case["every"])
        return s
    s["ctx"] = mhd.Context(nx, ny, dx, dy, case["eta"], courant=COURANT, safety=SAFETY,
                           ct_mode=mhd.CT_TRUE_ABS if case.get("true_abs") else mhd.CT_REFERENCE)
    u0 = _vortex(nx, ny, dx, dy, seed)
    if kind == "host":
        s["u0"] = u0.cpu().pin_memory()
        s["out"] = torch.empty_like(s["u0"]).pin_memory()
    elif kind == "rate":
        s["u0"], s["out"] = u0[4:].contiguous(), torch.empty_like(u0[4:])
    else:
        s["u0"], s["out"] = u0, torch.empty_like(u0)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        b = s["batch"]
        for i, u in enumerate(s["u0"]):
            b.set_state_device(i, _ptrs(u))
        b.run(case["steps"], record=False)
        for i, o in enumerate(s["out"]):
            b.get_state_device(i, _ptrs(o))
        return s["all"]
    if kind == "grad":
        u0 = s["u0"].detach().requires_grad_(True)
        eta = s["eta"].detach().requires_grad_(True)
        uT = mhd_autograd.trajectory(u0, eta, s["adj"])
        (0.5 * ((uT - s["target"]) ** 2).sum()).backward()
        return {"uT": uT.detach(), "g_u0": u0.grad, "g_eta": eta.grad}
    ctx = s["ctx"]
    if kind == "host":
        ctx.set_state(list(s["u0"].numpy()))
        ctx.step(0.0)  # the CFL step, chosen on the device
        ctx.get_state_into(list(s["out"].numpy()))
        return s["out"]
    if kind == "rate":
        dx, dy = _spacing(case)
        u, o = _ptrs(s["u0"]), _ptrs(s["out"])
        ctx.resistive_rate(u[0], u[1], o[0], o[1], solve_implicitly=True,
                           alpha=case["alpha_h2"] * min(dx, dy) ** 2)
        return s["out"]
    ctx.set_state_device(_ptrs(s["u0"]))
    dts = None
    if kind == "driver":
        dts = []
        for _ in range(case["steps"]):
            dt = ctx.cfl_dt()
            ctx.step(dt)
            dts.append(dt)
    else:
        ctx.run(case["steps"], dt_fixed=case.get("dt", 0.0), record=False)
    ctx.get_state_device(_ptrs(s["out"]))
    return {"u": s["out"]} if dts is None else {"u": s["out"], "dt": torch.tensor(dts, dtype=torch.float64)}


def work(case):
    """A step reads and writes the six planes (its CFL step needs the whole state before it, so two
    steps cannot share a read) and evaluates the explicit rate twice, about 700 operations a zone."""
    kind = case["kind"]
    if kind == "batch":
        zones = sum(n * n for n, _, _ in _ensemble(case, 0))
    else:
        zones = case["nx"] * case["ny"]
    if kind == "rate":
        return {"bytes": 32.0 * zones, "flops": 25.0 * zones}
    if kind == "grad":  # forward, and the adjoint step with its state, adjoint in and adjoint out
        return {"bytes": (96.0 + 144.0) * zones * case["steps"], "flops": 5600.0 * zones * case["steps"]}
    return {"bytes": 96.0 * zones * case["steps"], "flops": 1500.0 * zones * case["steps"]}


# ------------------------------------------------------------------------------------- exact
# The scheme in plain torch, 64 bits: MUSCL-minmod, HLL, upwind CT, ARS(2,2,2), with the implicit
# solves done exactly by FFT.


def _xp(f):
    return torch.roll(f, -1, -1)


def _xm(f):
    return torch.roll(f, 1, -1)


def _yp(f):
    return torch.roll(f, -1, -2)


def _ym(f):
    return torch.roll(f, 1, -2)


def _floor(f, lo):
    return torch.where(f < lo, torch.full_like(f, lo), f)


def _prims(U):
    rho0, mx, my, E, bx, by = U
    bxc, byc = (bx + _xp(bx)) / 2, (by + _yp(by)) / 2
    vx, vy = mx / rho0, my / rho0
    rho = _floor(rho0, 1e-8)
    p = _floor((GAMMA - 1) * (E - 0.5 * rho * (vx * vx + vy * vy) - (bxc * bxc + byc * byc) / 2), 1e-8)
    return rho, vx, vy, p, bxc, byc


def _faces(q, fwd, bwd):
    """States on the upper face of each cell: (this cell's upper value, the next cell's lower one)."""
    a, b = q - bwd(q), fwd(q) - q
    s = torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))
    return q + 0.5 * s, fwd(q - 0.5 * s)


def _flux_of(rho, vn, vt, p, bn, bt):
    """(mass, normal and tangential momentum, energy, tangential induction) flux, conserved state, fast speed."""
    b2, v2 = bn * bn + bt * bt, vn * vn + vt * vt
    pt = p + 0.5 * b2
    E = p / (GAMMA - 1) + 0.5 * (rho * v2 + b2)
    F = (rho * vn, rho * vn * vn + pt - bn * bn, rho * vn * vt - bn * bt,
         (E + pt) * vn - bn * (vn * bn + vt * bt), vn * bt - vt * bn)
    a2, t2, n2 = GAMMA * p / rho, b2 / rho, bn * bn / rho
    term = (t2 + a2) ** 2 - 4 * a2 * n2
    pos = term > 0
    sq = torch.where(pos, torch.sqrt(torch.where(pos, term, torch.ones_like(term))), torch.zeros_like(term))
    return F, (rho, rho * vn, rho * vt, E, bt), torch.sqrt(0.5 * (t2 + a2 + sq))


def _hll(L, R, bn):
    FL, UL, cL = _flux_of(*L[:4], bn, L[4])
    FR, UR, cR = _flux_of(*R[:4], bn, R[4])
    sL, sR = torch.minimum(L[1] - cL, R[1] - cR), torch.maximum(L[1] + cL, R[1] + cR)
    inv = 1.0 / torch.where(sR != sL, sR - sL, torch.ones_like(sL))
    return [torch.where(sL >= 0, fl, torch.where(sR <= 0, fr, (sR * fl - sL * fr + sL * sR * (ur - ul)) * inv))
            for fl, fr, ul, ur in zip(FL, FR, UL, UR)]


def _averaged(v, true_abs):
    return v.abs() < 1e-12 if true_abs else ~((v.abs() >= 1.0) & (v.abs() < 2147483648.0))


def _rates(U, dx, dy, true_abs):
    rho, vx, vy, p, bxc, byc = _prims(U)
    f = [_faces(q, _xp, _xm) for q in (rho, vx, vy, p, byc)]
    X = _hll([a for a, _ in f], [b for _, b in f], _xp(U[4]))  # mass, mx, my, E, by
    f = [_faces(q, _yp, _ym) for q in (rho, vy, vx, p, bxc)]
    Y = _hll([a for a, _ in f], [b for _, b in f], _yp(U[5]))  # mass, my, mx, E, bx
    Y = [Y[0], Y[2], Y[1], Y[3], Y[4]]
    eN, eS, eE, eW = -_xm(X[4]), -_xm(_ym(X[4])), _ym(Y[4]), _xm(_ym(Y[4]))
    corner = lambda q: 0.25 * (q + _xm(q) + _ym(q) + _xm(_ym(q)))  # noqa: E731
    vxc, vyc = corner(vx), corner(vy)
    ezy = torch.where(_averaged(vyc, true_abs), 0.5 * (eS + eN), torch.where(vyc > 0, eS, eN))
    ezx = torch.where(_averaged(vxc, true_abs), 0.5 * (eE + eW), torch.where(vxc > 0, eW, eE))
    ez = 0.5 * (ezx + ezy)
    R = [-((X[q] - _xm(X[q])) / dx + (Y[q] - _ym(Y[q])) / dy) for q in range(4)]
    return R + [-(_yp(ez) - ez) / dy, (_xp(ez) - ez) / dx]


def _current(bx, by, dx, dy):
    return (by - _xm(by)) / dx - (bx - _ym(bx)) / dy


def _curl(E, dx, dy):
    return -(_yp(E) - E) / dy, (_xp(E) - E) / dx


def _resistive(bx, by, eta, alpha, dx, dy):
    """Explicit (alpha None) or implicit rate of the face field."""
    b = eta * _current(bx, by, dx, dy)
    if alpha is not None:
        ny, nx = b.shape
        kx = 2 * math.pi * torch.arange(nx // 2 + 1, device=b.device, dtype=torch.float64) / nx
        ky = 2 * math.pi * torch.arange(ny, device=b.device, dtype=torch.float64) / ny
        # 4 sin^2(k/2) = 2 (1 - cos k), without its cancellation
        lam = (4 * torch.sin(kx / 2) ** 2)[None, :] / dx ** 2 + (4 * torch.sin(ky / 2) ** 2)[:, None] / dy ** 2
        b = torch.fft.irfft2(torch.fft.rfft2(b) / (1 + alpha * lam), s=(ny, nx))
    return _curl(b, dx, dy)


def _step(U, dt, eta, dx, dy, true_abs=False):
    g, d, alpha = ARS_G, ARS_D, dt * eta * ARS_G
    f1 = _rates(U, dx, dy, true_abs)
    S = [_floor(U[0], 1e-8)] + list(U[1:])
    u1 = [U[k] + f1[k] * (dt * g) for k in range(6)]
    u1[0] = _floor(u1[0], 1e-8)
    sx, sy = _resistive(u1[4], u1[5], eta, alpha, dx, dy)
    u1[4], u1[5] = u1[4] + sx * (dt * g), u1[5] + sy * (dt * g)
    f2 = _rates(u1, dx, dy, true_abs)
    gx, gy = _resistive(u1[4], u1[5], eta, None, dx, dy)
    a = [S[k] + f1[k] * (dt * d) + f2[k] * (dt * (1 - d)) for k in range(6)]
    a[4], a[5] = a[4] + gx * (dt * (1 - g)), a[5] + gy * (dt * (1 - g))
    sx, sy = _resistive(a[4], a[5], eta, alpha, dx, dy)
    gx, gy = _resistive(a[4] + sx * (dt * g), a[5] + sy * (dt * g), eta, None, dx, dy)
    return [_floor(a[0], 1e-8), a[1], a[2], a[3], a[4] + gx * (dt * g), a[5] + gy * (dt * g)]


def _cfl(U, eta, dx, dy):
    rho, vx, vy, p, bxc, byc = _prims(U)
    speed = torch.sqrt(GAMMA * p / rho + (bxc * bxc + byc * byc) / rho) + torch.sqrt(vx * vx + vy * vy)
    h = min(dx, dy)
    dt = COURANT * h / max(float(speed.max()), 1e-8)
    return SAFETY * (min(dt, h * h / (4 * eta)) if eta else dt)


def _advance(u0, case, dx, dy, eta, steps, dt=0.0):
    U, dts = [u0[k] for k in range(6)], []
    for _ in range(steps):
        dts.append(dt or _cfl(U, eta, dx, dy))
        U = _step(U, dts[-1], eta, dx, dy, bool(case.get("true_abs")))
    return torch.stack(U), dts


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for n, eta, sd in _ensemble(case, seed):
            h = 2 * math.pi / n
            out.append(_advance(_member(n, n, h, h, sd), case, h, h, eta, case["steps"])[0].reshape(-1))
        return torch.cat(out)
    nx, ny = case["nx"], case["ny"]
    dx, dy = _spacing(case)
    if kind == "grad":
        u0, target = _smooth(nx, ny, dx, dy, seed)
        u0.requires_grad_(True)
        eta = torch.tensor(case["eta"], dtype=torch.float64, device=u0.device, requires_grad=True)

        def one(U, e):
            return torch.stack(_step([U[k] for k in range(6)], case["dt"], e, dx, dy))

        U = u0
        for _ in range(case["steps"]):
            U = torch.utils.checkpoint.checkpoint(one, U, eta, use_reentrant=False)
        (0.5 * ((U - target) ** 2).sum()).backward()
        return {"uT": U.detach(), "g_u0": u0.grad, "g_eta": eta.grad}
    u0 = _vortex(nx, ny, dx, dy, seed)
    if kind == "rate":
        return torch.stack(_resistive(u0[4], u0[5], case["eta"], case["alpha_h2"] * min(dx, dy) ** 2, dx, dy))
    u, dts = _advance(u0, case, dx, dy, case["eta"], case["steps"], case.get("dt", 0.0))
    if kind == "driver":
        return {"u": u, "dt": torch.tensor(dts, dtype=torch.float64)}
    return u if kind == "host" else {"u": u}
