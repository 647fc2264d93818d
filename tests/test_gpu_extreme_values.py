"""Cells of no ordinary size -- a zero density, infinities, NaN, values whose squares overflow -- against the CPU
oracle, which works in plain IEEE operations: what is finite there is finite here, an infinite signal speed is
infinite (a CFL step of 0), and one cell's NaN reaches the cells that it reaches there.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps

# conserved values put into one cell of a uniform state (rho, mx, my, E, bxf, byf = 1, 0, 0, 1.5, 0.1, 0.2)
CELLS = {
    "no density": {0: 0.0, 1: 1.0, 2: -2.0},
    "square of the velocity overflows": {1: 1e200},
    "infinite energy": {3: np.inf},
    "square of the field overflows": {4: 1e200},
    "infinite density": {0: np.inf},
    "NaN density": {0: np.nan},
    "NaN energy": {3: np.nan},
    "large pressure": {3: 1e250},
    "large density and pressure": {0: 1e180, 3: 1e300},
    "small density": {0: 1e-200, 1: 1e-150},
}


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def _uniform(nx, ny, edit):
    u = [np.full((ny, nx), v) for v in (1.0, 0.0, 0.0, 1.5, 0.1, 0.2)]
    for k, v in edit.items():
        u[k][ny // 2, nx // 2] = v
    return u


@pytest.mark.parametrize("cell", CELLS)
@pytest.mark.parametrize("shape", [(12, 10), (300, 40)])
def test_cfl_and_primitives_of_any_cell(m, shape, cell):
    """Every entry that scans a state. A handful of operations a value: 16 eps relative."""
    import torch

    from oracle.oracle import Oracle

    nx, ny = shape
    dx, dy = 0.1, 0.07
    u = _uniform(nx, ny, CELLS[cell])
    orc = Oracle(nx, ny, dx, dy, 0.0)
    orc.set_state(u)
    want = orc.cfl_dt()
    ctx = m.Context(nx, ny, dx, dy, 0.0)
    batch = m.Batch([{"nx": nx, "ny": ny, "dx": dx, "dy": dy, "eta": 0.0}])
    dev = torch.tensor(np.stack(u), device="cuda")
    ptrs = [dev[k].data_ptr() for k in range(6)]
    torch.cuda.synchronize()
    got = []
    ctx.set_state(u)
    got.append(ctx.cfl_dt())
    prim = ctx.primitives()
    ctx.set_state_device(ptrs)
    got.append(ctx.cfl_dt())
    batch.set_state(0, u)
    got.append(batch.cfl_dt(0))
    batch.set_state_device(0, ptrs)
    got.append(batch.cfl_dt(0))
    assert all(abs(g - want) <= 16 * EPS * want for g in got), (got, want)
    for k, (name, w) in enumerate(orc.primitives().items()):
        g = prim[name] if isinstance(prim, dict) else prim[k]
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w)), name
        f = np.isfinite(w)
        assert np.all(np.abs(g[f] - w[f]) <= 16 * EPS * np.abs(w[f])), name
        assert np.array_equal(np.sign(g[np.isinf(w)]), np.sign(w[np.isinf(w)])), name
    ctx.close()
    batch.close()


def _modes(rng, nx, ny, amp):
    x, y = 2 * np.pi * np.arange(nx) / nx, 2 * np.pi * np.arange(ny) / ny
    f = np.zeros((ny, nx))
    for kx, ky in ((1, 0), (0, 1), (1, 1), (2, -1)):
        f += amp * rng.uniform(0.5, 1.0) * np.sin(kx * x[None, :] + ky * y[:, None] + rng.uniform(0, 6))
    return f


def _flow(nx, ny, dx, dy, v0, seed, rho=1.0, v=1.0):
    """A smooth flow in units of rho and v (pressure and field energy in rho v^2)."""
    rng = np.random.default_rng(seed)
    m = [_modes(rng, nx, ny, a) for a in (0.05, 0.03, 0.1, 0.1, 0.2)]
    r, p, vx, vy, az = 1 + m[0], 0.6 + m[1], v0[0] + m[2], v0[1] + m[3], m[4]
    bx, by = (np.roll(az, -1, 0) - az) / dy, -(np.roll(az, -1, 1) - az) / dx
    bxc, byc = 0.5 * (bx + np.roll(bx, -1, 1)), 0.5 * (by + np.roll(by, -1, 0))
    E = p / (5.0 / 3.0 - 1) + 0.5 * r * (vx * vx + vy * vy) + 0.5 * (bxc * bxc + byc * byc)
    b = np.sqrt(rho) * v
    return [np.ascontiguousarray(f) for f in (rho * r, rho * v * r * vx, rho * v * r * vy, rho * v * v * E, b * bx, b * by)]


@pytest.mark.parametrize("rho,v", [(1e90, 1e35), (1e200, 1e-25), (1e20, 1e70), (1e70, 1.0)])
@pytest.mark.parametrize("v0", [(0.0, 0.0), (6.0, 0.2), (-5.0, 6.0)])
def test_step_in_far_units(m, rho, v, v0):
    """States whose pressure, field energy or products with the density are beyond what the straight-line fluxes
    take, but well within the quotients' range: two steps against the oracle, at the single-step tolerance of the
    parity tests (1e-12 relative L-infinity a field)."""
    from oracle.oracle import Oracle

    nx, ny = 57, 31
    dx, dy = 2 * np.pi / nx, 1.4 * np.pi / ny
    eta = 0.01 * v
    ic = _flow(nx, ny, dx, dy, v0, 7, rho, v)
    orc = Oracle(nx, ny, dx, dy, eta)
    orc.set_state(ic)
    ctx = m.Context(nx, ny, dx, dy, eta)
    ctx.set_state(ic)
    batch = m.Batch([{"nx": nx, "ny": ny, "dx": dx, "dy": dy, "eta": eta}])
    batch.set_state(0, ic)
    for _ in range(2):
        dt = 0.5 * orc.cfl_dt()
        assert abs(0.5 * ctx.cfl_dt() - dt) <= 1e-13 * dt
        orc.step(dt)
        ctx.step(dt)
        batch.step([dt])
    assert ctx.synchronize_status() == 0 and batch.synchronize_status()[0] == 0
    for g, h, w in zip(ctx.get_state(), batch.get_state(0), orc.get_state()):
        assert np.abs(g - w).max() <= 1e-12 * np.abs(w).max()
        assert np.abs(h - w).max() <= 1e-12 * np.abs(w).max()
    ctx.close()
    batch.close()


BAD = {"NaN energy": {3: np.nan}, "infinite energy": {3: np.inf}, "infinite momentum": {1: np.inf},
       "no density": {0: 0.0, 1: 1.0}, "NaN field": {4: np.nan}}


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("at", [(0, 0), (27, 2), (28, 16), (56, 30), (40, 11)])
@pytest.mark.parametrize("v0", [(0.0, 0.0), (6.0, 0.2), (-5.0, 6.0)])
def test_one_bad_cell_reaches_the_cells_it_reaches_in_the_oracle(m, at, bad, v0):
    """An ideal step (eta = 0, its solves give 0) of a state with one such cell, at strip and segment edges: the
    cells that it makes non-finite are those of the scheme in IEEE operations, the others keep their values."""
    from oracle.oracle import Oracle

    nx, ny = 57, 31
    dx, dy = 2 * np.pi / nx, 1.4 * np.pi / ny
    ic = _flow(nx, ny, dx, dy, v0, 9)
    dt = 1e-3
    for k, val in BAD[bad].items():
        ic[k][at[1], at[0]] = val
    orc = Oracle(nx, ny, dx, dy, 0.0)

    def rate(u):
        orc.set_state(u)
        return orc.explicit_rhs()

    g = m.ars_gamma()
    d = 1 - 1 / (2 * g)
    with np.errstate(all="ignore"):
        f1 = rate(ic)
        u1 = [u + dt * g * f for u, f in zip(ic, f1)]
        f2 = rate([np.where(u1[0] < 1e-8, 1e-8, u1[0])] + u1[1:])
        want = [u + dt * d * a + dt * (1 - d) * b for u, a, b in zip(ic, f1, f2)]
        # the resistive terms are 0 times the current of a field that may not be finite
        for b in (u1, want):
            e = 0.0 * ((b[5] - np.roll(b[5], 1, 1)) - (b[4] - np.roll(b[4], 1, 0)))
            want[4], want[5] = want[4] - (np.roll(e, -1, 0) - e), want[5] + (np.roll(e, -1, 1) - e)
    ctx = m.Context(nx, ny, dx, dy, 0.0)
    ctx.set_state(ic)
    ctx.step(dt)
    assert ctx.synchronize_status() == 3  # MHD_ERR_NONFINITE
    for k, (got, w) in enumerate(zip(ctx.get_state(), want)):
        fin = np.isfinite(w)
        assert np.array_equal(np.isfinite(got), fin), (k, np.argwhere(np.isfinite(got) != fin)[:8])
        assert np.abs(got[fin] - w[fin]).max() <= 1e-12 * max(np.abs(w[fin]).max(), 1.0), k
    ctx.close()


@pytest.mark.parametrize("rho,v", [(1e90, 1e35), (1e200, 1e-25), (1e20, 1e70), (1.0, 1.0)])
@pytest.mark.parametrize("v0", [(0.0, 0.0), (6.0, 0.2), (-5.0, 6.0)])
def test_rate_vjp_in_far_units(m, rho, v, v0):
    """The explicit rate's VJP of such states against PyTorch autograd through the restated rate, at the suite's
    bound for these quantities (1e-9 relative a field)."""
    import torch

    from oracle import torch_step as ts

    nx, ny = 53, 17
    dx, dy = 2 * np.pi / nx, 1.4 * np.pi / ny
    U = torch.tensor(np.stack(_flow(nx, ny, dx, dy, v0, 7, rho, v)))
    # an adjoint in the inverse units of the rates, so that every rate counts alike
    unit = torch.tensor([rho, rho * v, rho * v, rho * v * v, np.sqrt(rho) * v, np.sqrt(rho) * v], dtype=torch.float64)
    w = torch.randn(6, ny, nx, generator=torch.Generator().manual_seed(5), dtype=torch.float64) / unit[:, None, None]
    Ut = [U[k].clone().requires_grad_(True) for k in range(6)]
    want = torch.autograd.grad(ts.explicit_rhs(Ut, dx, dy), Ut, grad_outputs=list(w))
    assert all(torch.isfinite(t).all() for t in want)
    adj = m.Adjoint(nx, ny, dx, dy, 1e-2, 1e-3, 1)
    u_d, w_d = U.cuda().contiguous(), w.cuda().contiguous()
    out = torch.empty_like(u_d)
    torch.cuda.synchronize()
    adj.rate_vjp([u_d[k].data_ptr() for k in range(6)], [w_d[k].data_ptr() for k in range(6)],
                 [out[k].data_ptr() for k in range(6)])
    for k in range(6):
        err = float((out[k].cpu() - want[k]).abs().max() / want[k].abs().max())
        assert err <= 1e-9, (k, err)
    adj.close()


# grids whose solves take the two passes, the chip's shared memory (t > 0.06) and, larger, the sweeps
@pytest.mark.parametrize("nx,ny,eta", [(300, 290, 1e-4), (300, 290, 0.5), (1300, 1000, 1e-4), (1300, 1000, 0.5)])
@pytest.mark.parametrize("dt", [0.0, 1e-4])
def test_solve_of_a_bad_field_is_reported(m, nx, ny, eta, dt):
    """A NaN in the field breaks every form of the solve down: the status says so, and the next state steps on."""
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    ic = m.problems.orszag_tang(nx, ny, dx, dy)
    bad = [f.copy() for f in ic]
    bad[4][ny // 3, nx // 2] = np.nan
    ctx = m.Context(nx, ny, dx, dy, eta)
    batch = m.Batch([{"nx": n, "ny": k, "dx": dx, "dy": dy, "eta": eta} for n, k in ((nx, ny), (nx, ny))])
    ctx.set_state(bad)
    batch.set_state(0, bad)
    batch.set_state(1, ic)
    ctx.step(dt)
    assert ctx.synchronize_status() == 3  # MHD_ERR_NONFINITE
    batch.step([dt, dt] if dt else None)
    worst, each = batch.synchronize_status()
    assert worst == 3 and list(each) == [3, 0]
    ctx.set_state(ic)
    ctx.step(dt)
    assert ctx.synchronize_status() == 0
    for g, w in zip(batch.get_state(1), ctx.get_state()):
        assert np.abs(g - w).max() <= 1e-12 * max(np.abs(w).max(), 1.0)
    ctx.close()
    batch.close()
