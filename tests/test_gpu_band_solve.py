"""The implicit solve with every vector in the chip's shared memory: one band of rows, two, one short of all SMs and
all of them, bands of even and uneven heights, one, two and four runs a thread, the widest grid that fits and the
first that does not. Reference and tolerance: those of test_gpu_solve_forms.py."""
import numpy as np
import pytest

from test_gpu_solve_forms import EPS, _cg, _faces, _rate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


@pytest.mark.parametrize("shape", [(2047, 2), (2048, 17), (2049, 17), (3, 12001), (190, 191), (401, 145), (333, 592),
                                   (511, 300), (513, 297), (1024, 299), (700, 741)])
@pytest.mark.parametrize("t,kind", [(4e-3, "smooth"), (0.3, "rough"), (4.0, "noise")])
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


@pytest.mark.parametrize("cap", [1, 2, 7])
def test_capped_solve_is_cgs_iterate(m, cap):
    nx, ny = 260, 250
    dx = dy = 2 * np.pi / nx
    alpha = 0.3 * dx * dx / 4
    bx, by = _faces(nx, ny, dx, dy, "noise", seed=3)
    gx, gy, prods, status = _rate(m, nx, ny, dx, dy, 0.7, alpha, bx, by, cg_max_iters=cap)
    x, k = _cg(bx, by, dx, dy, 0.7, alpha, max_iters=cap)
    assert prods == k == cap and status == 4  # MHD_ERR_CG_NOT_CONVERGED
    bound = 64 * EPS * np.abs(x).max() / dx
    assert np.abs(gx + (np.roll(x, -1, 0) - x) / dy).max() <= bound
    assert np.abs(gy - (np.roll(x, -1, 1) - x) / dx).max() <= bound


def test_step_chosen_on_the_device_or_by_the_caller(m):
    """The CFL step's solves come behind the two-pass form, those of a given dt alone: the same bits."""
    from tests_helpers import smooth_state

    nx, ny = 301, 230
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    ic = smooth_state(nx, ny, dx, dy, 5, v_amp=0.3)
    ctx, fixed = m.Context(nx, ny, dx, dy, 0.3), m.Context(nx, ny, dx, dy, 0.3)
    for c in (ctx, fixed):
        c.set_state(ic)
    for _ in range(3):
        dt = ctx.cfl_dt()
        assert 2 * dt * m.ars_gamma() * 0.3 * (1 / dx**2 + 1 / dy**2) > 0.06
        ctx.step(0.0)
        fixed.step(dt)
        assert ctx.last_cg_products() == fixed.last_cg_products()
    for a, b in zip(ctx.get_state(), fixed.get_state()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("t,kind,few", [(0.05, "noise", False), (0.05, "smooth", True), (0.03, "noise", True)])
def test_step_on_either_side_of_the_two_pass_forms_range(m, t, kind, few):
    """A grid that the chip holds, with t where the two passes' levels may not suffice: a CFL step and a step of that
    dt take the same kernels from there on, and below (0.03) the passes settle even noise in nine products."""
    nx, ny = 301, 230
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    ic = m.problems.orszag_tang(nx, ny, dx, dy)
    bx, by = _faces(nx, ny, dx, dy, kind, seed=2)
    for k, b in ((4, bx), (5, by)):
        ic[k] = ic[k] + 0.2 * b / max(np.abs(bx).max(), np.abs(by).max())
    probe = m.Context(nx, ny, dx, dy, 0.0)
    probe.set_state(ic)
    eta = t / (2 * (1 / dx**2 + 1 / dy**2)) / (probe.cfl_dt() * m.ars_gamma())
    a, b = m.Context(nx, ny, dx, dy, eta), m.Context(nx, ny, dx, dy, eta)
    for c in (a, b):
        c.set_state(ic)
    dt = a.cfl_dt()
    a.step(0.0)
    b.step(dt)
    assert a.synchronize_status() == b.synchronize_status() == 0
    assert a.last_cg_products() == b.last_cg_products()
    assert (max(a.last_cg_products()) <= 9) == few
    for u, v in zip(a.get_state(), b.get_state()):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("shape", [(682, 888), (683, 888), (512, 512), (520, 521), (1365, 290), (1024, 592), (1025, 592)])
def test_rate_on_half_the_chip_and_on_all_of_it(m, shape):
    """The largest grids whose bands fit half of the SMs, and the next ones (four and two runs a thread)."""
    nx, ny = shape
    dx, dy, eta = 2 * np.pi / nx, 1.3 * 2 * np.pi / ny, 0.7
    alpha = 0.3 / (2 * (1 / dx**2 + 1 / dy**2))
    bx, by = _faces(nx, ny, dx, dy, "noise", seed=nx * 31 + ny)
    gx, gy, prods, status = _rate(m, nx, ny, dx, dy, eta, alpha, bx, by)
    x, k = _cg(bx, by, dx, dy, eta, alpha)
    assert status == 0
    assert abs(prods - k) <= 1, (prods, k)
    bound = 64 * EPS * np.abs(x).max() / min(dx, dy)
    assert np.abs(gx + (np.roll(x, -1, 0) - x) / dy).max() <= bound
    assert np.abs(gy - (np.roll(x, -1, 1) - x) / dx).max() <= bound
