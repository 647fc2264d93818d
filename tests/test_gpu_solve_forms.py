"""The implicit solve's forms -- one cluster with everything in shared memory, two passes from moments,
the ordinary CG sweeps, and the hand-over from one to the other -- at the sizes where their strips, bands
and segments end, through mhd_resistive_rate and mhd_step.

Reference: plain numpy CG (x0 = 0, constant Jacobi diagonal, stop when |r|^2 < eps^2 |b|^2: the
reference's solver, solvers.hpp:404-489 with Eigen's defaults) on the same right-hand side. Both
solutions have a residual of eps |b|, and rounding adds a few eps |x|: 16 eps |x|_max each is allowed,
which the rate's difference quotients turn into 2 * 2 * 16 eps |x|_max / h. Products may differ by one
(a residual at the threshold).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
TOL = 2.0 ** -52  # the library's default tolerance


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def _faces(nx, ny, dx, dy, kind, seed):
    """Divergence-free face field: a few modes ("smooth"), with a little noise ("rough"), or noise."""
    rng = np.random.default_rng(seed)
    x, y = np.arange(nx) * 2 * np.pi / nx, np.arange(ny) * 2 * np.pi / ny
    az = np.zeros((ny, nx))
    if kind != "noise":
        for kx, ky in ((1, 0), (0, 1), (2, 1), (1, 3)):
            az += rng.uniform(0.2, 1.0) * np.sin(kx * x[None, :] + ky * y[:, None] + rng.uniform(0, 6))
    az += {"smooth": 0.0, "rough": 1e-4, "noise": 1.0}[kind] * rng.standard_normal((ny, nx))
    return (np.roll(az, -1, 0) - az) / dy, -(np.roll(az, -1, 1) - az) / dx


def _cg(bx, by, dx, dy, eta, alpha, max_iters=10**6):
    cx, cy = alpha / dx**2, alpha / dy**2
    d = 1 + 2 * (cx + cy)
    b = eta * ((by - np.roll(by, 1, 1)) / dx - (bx - np.roll(bx, 1, 0)) / dy)

    def A(p):
        return d * p - cx * (np.roll(p, 1, 1) + np.roll(p, -1, 1)) - cy * (np.roll(p, 1, 0) + np.roll(p, -1, 0))

    x, r, p = np.zeros_like(b), b.copy(), b / d
    rz, thr, k = (r * p).sum(), max(TOL**2 * (b * b).sum(), np.finfo(float).tiny), 0
    if not (b * b).sum() >= thr:
        return x, 0
    while k < max_iters:
        q = A(p)
        a = rz / (p * q).sum()
        x, r, k = x + a * p, r - a * q, k + 1
        if (r * r).sum() < thr:
            break
        rz, old = (r * r / d).sum(), rz
        p = r / d + rz / old * p
    return x, k


def _rate(m, nx, ny, dx, dy, eta, alpha, bx, by, **kw):
    import torch

    ctx = m.Context(nx, ny, dx, dy, eta, **kw)
    dbx, dby = torch.tensor(bx, device="cuda"), torch.tensor(by, device="cuda")
    ox, oy = torch.empty_like(dbx), torch.empty_like(dby)
    torch.cuda.synchronize()
    prods = ctx.resistive_rate(dbx.data_ptr(), dby.data_ptr(), ox.data_ptr(), oy.data_ptr(), solve_implicitly=True,
                               alpha=alpha)
    status = ctx.synchronize_status()
    ctx.close()
    return ox.cpu().numpy(), oy.cpu().numpy(), prods, status


# clusters of 1 .. 8 blocks with bands of one row and more, one cell or runs of four rows a thread, odd
# widths, the largest that fits (181 x 181) and the first that does not; a grid for the sweeps
@pytest.mark.parametrize("shape", [(2, 2), (3, 5), (78, 4), (79, 9), (84, 33), (85, 64), (1021, 8), (157, 131), (181, 181),
                                   (182, 181), (300, 290)])
@pytest.mark.parametrize("t,kind", [(4e-4, "smooth"), (4e-4, "noise"), (8e-3, "rough"), (1.4e-2, "noise"), (4e-2, "rough"),
                                    (5.5e-2, "noise"), (0.3, "rough"), (2.0, "noise")])
def test_rate_matches_plain_cg(m, shape, t, kind):
    nx, ny = shape
    dx, dy, eta = 2 * np.pi / nx, 1.3 * 2 * np.pi / ny, 0.7
    alpha = t / (2 * (1 / dx**2 + 1 / dy**2))
    bx, by = _faces(nx, ny, dx, dy, kind, seed=nx * 31 + ny)
    gx, gy, prods, status = _rate(m, nx, ny, dx, dy, eta, alpha, bx, by)
    x, k = _cg(bx, by, dx, dy, eta, alpha)
    assert status == 0
    assert abs(prods - k) <= 1, (prods, k)
    bound = 64 * EPS * np.abs(x).max() / min(dx, dy)
    assert np.abs(gx + (np.roll(x, -1, 0) - x) / dy).max() <= bound
    assert np.abs(gy - (np.roll(x, -1, 1) - x) / dx).max() <= bound


@pytest.mark.parametrize("t,cap", [(8e-3, 1), (8e-3, 3), (4e-2, 4), (0.3, 3)])
def test_capped_solve_is_cgs_iterate(m, t, cap):
    """A solve stopped by its cap returns that CG iterate and says so, in either form."""
    nx, ny = 90, 70
    dx = dy = 2 * np.pi / nx
    alpha = t * dx * dx / 4
    bx, by = _faces(nx, ny, dx, dy, "noise", seed=3)
    gx, gy, prods, status = _rate(m, nx, ny, dx, dy, 0.7, alpha, bx, by, cg_max_iters=cap)
    x, k = _cg(bx, by, dx, dy, 0.7, alpha, max_iters=cap)
    assert prods == k == cap and status == 4  # MHD_ERR_CG_NOT_CONVERGED
    bound = 64 * EPS * np.abs(x).max() / dx
    assert np.abs(gx + (np.roll(x, -1, 0) - x) / dy).max() <= bound
    assert np.abs(gy - (np.roll(x, -1, 1) - x) / dx).max() <= bound


def test_loose_tolerance_stops_early(m):
    nx, ny = 120, 60
    dx = dy = 2 * np.pi / nx
    bx, by = _faces(nx, ny, dx, dy, "noise", seed=4)
    few = _rate(m, nx, ny, dx, dy, 0.7, 1e-2 * dx * dx / 4, bx, by, cg_tol=1e-6)
    full = _rate(m, nx, ny, dx, dy, 0.7, 1e-2 * dx * dx / 4, bx, by)
    assert few[3] == full[3] == 0 and 0 < few[2] < full[2]
    # |r| < 1e-6 |b| and the matrix's smallest eigenvalue is 1
    assert np.linalg.norm(few[0] - full[0]) <= 1e-5 * np.linalg.norm(full[0])


# the moment form through a step of fixed dt (U* = U where nothing moves: rho = p = 1, v = 0 and a field so
# weak that the explicit stage leaves its faces alone to rounding): widths below, at and above a strip's
# output columns (84, 78 with three columns a lane; 22, 18, 14 with one), t in each variant's range
@pytest.mark.parametrize("shape", [(234, 200), (235, 211), (252, 180), (253, 190), (700, 61), (1030, 47), (1500, 260)])
@pytest.mark.parametrize("t,kind", [(4e-4, "smooth"), (8e-3, "rough"), (1.4e-2, "noise"), (4e-2, "rough"), (5.5e-2, "noise")])
def test_step_in_moment_form_matches_plain_cg(m, shape, t, kind):
    nx, ny = shape
    dx, dy = 2 * np.pi / nx, 1.3 * 2 * np.pi / ny
    dt = 1e-9
    g = m.ars_gamma()
    eta = t / (2 * (1 / dx**2 + 1 / dy**2)) / (dt * g)
    bx, by = _faces(nx, ny, dx, dy, kind, seed=nx * 31 + ny)
    scale = 1e-6 / max(np.abs(bx).max(), np.abs(by).max())
    bx, by = scale * bx, scale * by
    one, zero = np.ones((ny, nx)), np.zeros((ny, nx))
    ctx = m.Context(nx, ny, dx, dy, eta)
    ctx.set_state([one, zero, zero, 1.5 * one, bx, by])
    ctx.step(dt)
    assert ctx.synchronize_status() == 0
    got, prods = ctx.get_state(), ctx.last_cg_products()
    ctx.close()
    # the step's linear part (solvers.hpp:491-613 without the explicit rates)
    alpha = dt * eta * g

    def curl(e):
        return -(np.roll(e, -1, 0) - e) / dy, (np.roll(e, -1, 1) - e) / dx

    def jz(u, v):
        return eta * ((v - np.roll(v, 1, 1)) / dx - (u - np.roll(u, 1, 0)) / dy)

    x1, k1 = _cg(bx, by, dx, dy, eta, alpha)
    r = curl(x1)
    b1 = bx + dt * g * r[0], by + dt * g * r[1]
    r = curl(jz(*b1))
    a = bx + dt * (1 - g) * r[0], by + dt * (1 - g) * r[1]
    x2, k2 = _cg(*a, dx, dy, eta, alpha)
    r = curl(x2)
    r = curl(jz(a[0] + dt * g * r[0], a[1] + dt * g * r[1]))
    want = a[0] + dt * g * r[0], a[1] + dt * g * r[1]
    assert abs(prods[0] - k1) <= 1 and abs(prods[1] - k2) <= 1, (prods, k1, k2)
    # the implicit increments dt g curl(x) are t |B| or less, known to 64 eps as in the rates above; sums and
    # the explicit stage (numerical diffusion dt c / h < 1e-6 of B's variation from cell to cell) on top
    bound = (64 * EPS + 2e-6 * dt * 2 * np.sqrt(5 / 3) / min(dx, dy) / 1e-6) * 1e-6 * 4
    assert max(np.abs(got[4] - want[0]).max(), np.abs(got[5] - want[1]).max()) <= bound


@pytest.mark.parametrize("t,noise", [(0.15, 0.0), (0.05, 0.3)])
def test_cfl_step_hands_the_solve_over(m, t, noise):
    """Above 256^2 a CFL step's solve starts in the moment form, which leaves it to the sweeps when the
    device's dt turns out too large (t = 0.15) or its levels do not suffice (a noisy field at t = 0.05).
    The same step with that dt given takes another route to the same state."""
    nx, ny = 300, 290
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    ic = m.problems.orszag_tang(nx, ny, dx, dy)
    rng = np.random.default_rng(8)
    az = noise * dx * rng.standard_normal((ny, nx))
    ic[4] += (np.roll(az, -1, 0) - az) / dy
    ic[5] -= (np.roll(az, -1, 1) - az) / dx
    probe = m.Context(nx, ny, dx, dy, 0.0)
    probe.set_state(ic)
    dt0 = probe.cfl_dt()
    eta = t / (2 * (1 / dx**2 + 1 / dy**2)) / (dt0 * m.ars_gamma())
    a, b = m.Context(nx, ny, dx, dy, eta), m.Context(nx, ny, dx, dy, eta)
    a.set_state(ic)
    b.set_state(ic)
    dt = a.cfl_dt()
    a.step(0.0)
    b.step(dt)
    assert a.synchronize_status() == b.synchronize_status() == 0
    assert all(abs(p - q) <= 1 for p, q in zip(a.last_cg_products(), b.last_cg_products()))
    assert max(a.last_cg_products()) > 9  # beyond the moment form's levels
    for u, v in zip(a.get_state(), b.get_state()):
        assert np.abs(u - v).max() <= 64 * EPS * max(np.abs(v).max(), 1.0) * (1 if noise == 0 else 4)
    for c in (probe, a, b):
        c.close()
