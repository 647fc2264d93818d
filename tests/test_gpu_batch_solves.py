"""The batch's solves by form: instances that take a cluster, the moment form, and the sweeps (what the moment
form leaves: a large t, more products than it resolves), mixed in one batch, and clusters of every size.
Each instance against a single context stepped with the same dt: the explicit stages are the same sweeps, so
the states differ by the solves' rounding only: 1e-12 relative L-infinity (the single-step tolerance of the
parity tests; fields below 1 against 1), products within one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _check(m, shapes, etas, steps=2, noise=0.0):
    specs, states = [], []
    for k, ((nx, ny), eta) in enumerate(zip(shapes, etas)):
        dx, dy = 2 * np.pi / nx, 2.2 * np.pi / ny
        ic = m.problems.orszag_tang(nx, ny, dx, dy)
        az = noise * dx * np.random.default_rng(k).standard_normal((ny, nx))
        ic[4] += (np.roll(az, -1, 0) - az) / dy
        ic[5] -= (np.roll(az, -1, 1) - az) / dx
        specs.append(dict(nx=nx, ny=ny, dx=dx, dy=dy, eta=eta))
        states.append(ic)
    b = m.Batch(specs)
    ctxs = [m.Context(s["nx"], s["ny"], s["dx"], s["dy"], s["eta"]) for s in specs]
    for i, ic in enumerate(states):
        b.set_state(i, ic)
        ctxs[i].set_state(ic)
    for _ in range(steps):
        dts = [c.cfl_dt() for c in ctxs]
        b.step()  # every instance's own CFL step, chosen on the device
        for c, dt in zip(ctxs, dts):
            c.step(dt)
    assert b.synchronize_status()[0] == 0
    prods = b.last_cg_products()
    for i, c in enumerate(ctxs):
        c.synchronize()
        assert np.abs(prods[i] - np.array(c.last_cg_products())).max() <= 1, (i, prods[i], c.last_cg_products())
        for g, w in zip(b.get_state(i), c.get_state()):
            assert np.abs(g - w).max() <= TOL * max(np.abs(w).max(), 1.0), i
        c.close()
    b.close()
    return prods


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def test_all_forms_in_one_batch(m):
    """Clusters, every level count of the moment form, a t beyond it, eta = 0, and widths on either side of
    the tiles' output columns (84, 78)."""
    shapes = [(64, 64), (2, 2), (5, 300), (234, 234), (235, 200), (252, 256), (253, 190), (400, 300), (300, 290), (320, 260)]
    etas = [1e-3, 1e-2, 5e-3, 1e-5, 3e-4, 1e-3, 4e-3, 6e-3, 2e-1, 0.0]
    prods = _check(m, shapes, etas)
    assert prods[8].min() > 9 and prods[9].max() == 0


def test_moment_form_leaves_noisy_fields_to_the_sweeps(m):
    _check(m, [(300, 280), (260, 300), (240, 240)], [9e-3, 9e-3, 1e-3], noise=0.4)


@pytest.mark.parametrize("count,n", [(3, 150), (20, 60), (40, 33), (150, 24), (9, 181)])
def test_clusters_of_every_size(m, count, n):
    _check(m, [(n, n + k % 3) for k in range(count)], [10 ** (-1 - 3 * (k % 7) / 6) for k in range(count)], steps=1)
