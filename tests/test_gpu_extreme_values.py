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
