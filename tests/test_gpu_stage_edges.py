"""The explicit stages and the finalize at the edges of their strips (28 columns) and row segments (3 rows
or more), and in every case of the HLL flux: subsonic, and supersonic to either side in x, in y and in
both (the clamped wave speeds' one-sided limits), against the CPU oracle. Two steps; the single-step
tolerance of the parity tests, 1e-12 relative L-infinity per field (fields below 1 against 1).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP_TOL = 1e-12


def _state(nx, ny, dx, dy, vx0, vy0, seed):
    rng = np.random.default_rng(seed)
    x, y = 2 * np.pi * np.arange(nx) / nx, 2 * np.pi * np.arange(ny) / ny

    def modes(amp):
        f = np.zeros((ny, nx))
        for kx, ky in ((1, 0), (0, 1), (1, 1), (2, -1)):
            f += amp * rng.uniform(0.5, 1.0) * np.sin(kx * x[None, :] + ky * y[:, None] + rng.uniform(0, 6))
        return f

    rho, p, vx, vy, az = 1 + modes(0.05), 0.6 + modes(0.03), vx0 + modes(0.1), vy0 + modes(0.1), modes(0.2)
    bx, by = (np.roll(az, -1, 0) - az) / dy, -(np.roll(az, -1, 1) - az) / dx
    bxc, byc = 0.5 * (bx + np.roll(bx, -1, 1)), 0.5 * (by + np.roll(by, -1, 0))
    E = p / (5.0 / 3.0 - 1) + 0.5 * rho * (vx * vx + vy * vy) + 0.5 * (bxc * bxc + byc * byc)
    return [np.ascontiguousarray(f) for f in (rho, rho * vx, rho * vy, E, bx, by)]


@pytest.mark.parametrize("shape", [(28, 3), (29, 4), (27, 5), (56, 7), (57, 10), (85, 31)])
@pytest.mark.parametrize("flow", [(0.0, 0.0), (6.0, 0.0), (-6.0, 0.3), (0.2, 7.0), (0.0, -7.0), (5.0, -6.0)])
def test_step_at_strip_and_segment_edges(shape, flow):
    import torch

    import magnetohydrodynamics_simulator_b200 as m
    from oracle.oracle import Oracle

    assert torch.cuda.is_available()
    nx, ny = shape
    dx, dy = 2 * np.pi / nx, 1.4 * np.pi / ny
    ic = _state(nx, ny, dx, dy, *flow, seed=nx * 100 + ny)
    orc = Oracle(nx, ny, dx, dy, 0.01)
    orc.set_state(ic)
    ctx = m.Context(nx, ny, dx, dy, 0.01)
    ctx.set_state(ic)
    for _ in range(2):
        dt = 0.5 * orc.cfl_dt()
        assert abs(0.5 * ctx.cfl_dt() - dt) <= 1e-13 * dt
        orc.step(dt)
        ctx.step(dt)
    ctx.synchronize()
    for g, w in zip(ctx.get_state(), orc.get_state()):
        assert np.abs(g - w).max() <= STEP_TOL * max(np.abs(w).max(), 1.0)
    ctx.close()
