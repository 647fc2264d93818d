"""The two-pass solve's solution itself, through resistive_rate on grids large enough that a caller's field takes it:
every level count, strips of whole, one more and one less output columns (84, 78 with three columns a lane; 22, 18,
14 with one), grids of few columns and of few rows, and the hand-over to the sweeps at t = 0.05.

Reference: the periodic matrix inverted by FFT in numpy, with one step of refinement (error about an eps of x). The
library's solution has a residual below eps |b| (2-norm; A >= 1, so |x|'s error is no larger), and a few eps of rounding
a level: 8 eps |x|_max is allowed, which the rate's difference quotients double.
"""
import numpy as np
import pytest

from test_gpu_solve_forms import EPS, TOL, _faces, _rate


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def _matrix(nx, ny, dx, dy, alpha):
    cx, cy = alpha / dx**2, alpha / dy**2
    d = 1 + 2 * (cx + cy)

    def A(p):
        return d * p - cx * (np.roll(p, 1, 1) + np.roll(p, -1, 1)) - cy * (np.roll(p, 1, 0) + np.roll(p, -1, 0))

    ex = 2 - 2 * np.cos(2 * np.pi * np.arange(nx // 2 + 1) / nx)
    ey = 2 - 2 * np.cos(2 * np.pi * np.arange(ny) / ny)
    return A, d, 1 + cx * ex[None, :] + cy * ey[:, None]


def _solve(b, A, eig):
    x = np.fft.irfft2(np.fft.rfft2(b) / eig, s=b.shape)
    return x + np.fft.irfft2(np.fft.rfft2(b - A(x)) / eig, s=b.shape)


def _products(b, A, d):
    """CG's products, and its second to last iterate."""
    x, r, p = np.zeros_like(b), b.copy(), b / d
    rz, thr, k, last = (r * p).sum(), TOL**2 * (b * b).sum(), 0, None
    while True:
        q = A(p)
        a = rz / (p * q).sum()
        last = x
        x, r, k = x + a * p, r - a * q, k + 1
        if (r * r).sum() < thr:
            return k, last
        rz, old = (r * r / d).sum(), rz
        p = r / d + rz / old * p


def _curl_error(gx, gy, x, dx, dy):
    """Error of the rate -curl x in units of x: difference quotients times the spacing."""
    ex = np.abs(gx * dy + (np.roll(x, -1, 0) - x)).max()
    ey = np.abs(gy * dx - (np.roll(x, -1, 1) - x)).max()
    return max(ex, ey)


# t and shapes by level count (5, 7, 9, and 9 with the sweeps behind)
CASES = [(8e-4, s) for s in ((2268, 2121), (2269, 2120), (2267, 2118), (31, 156001), (160001, 30))]
CASES += [(1e-2, s) for s in ((1560, 1400), (1561, 1399), (1559, 1351), (1448, 1449), (18, 120001), (37, 60000), (70001, 31))]
CASES += [(0.02, s) for s in ((1872, 1560), (1873, 1553), (1871, 1551), (28, 104000), (97001, 30), (5000, 601))]
CASES += [(0.05, s) for s in ((1873, 1553), (1716, 1700), (97001, 30))]


@pytest.mark.gpu
@pytest.mark.parametrize("t,shape", CASES)
@pytest.mark.parametrize("kind", ["smooth", "noise"])
def test_solution(m, t, shape, kind):
    nx, ny = shape
    dx, dy, eta = 2 * np.pi / nx, 1.3 * 2 * np.pi / ny, 0.7
    alpha = t / (2 * (1 / dx**2 + 1 / dy**2))
    bx, by = _faces(nx, ny, dx, dy, kind, seed=nx + 3 * ny)
    gx, gy, prods, status = _rate(m, nx, ny, dx, dy, eta, alpha, bx, by)
    assert status == 0
    b = eta * ((by - np.roll(by, 1, 1)) / dx - (bx - np.roll(bx, 1, 0)) / dy)
    A, d, eig = _matrix(nx, ny, dx, dy, alpha)
    x = _solve(b, A, eig)
    assert _curl_error(gx, gy, x, dx, dy) <= 16 * EPS * np.abs(x).max()
    if kind == "noise":
        assert prods == {8e-4: 5, 1e-2: 7, 0.02: 8, 0.05: 10}[t]


@pytest.mark.parametrize("t,shape", [(8e-4, (2269, 2120)), (1e-2, (1561, 1399)), (0.02, (1873, 1553))])
def test_one_product_less_would_not_do(t, shape):
    """The bound above, on the CPU: CG's iterate one product short fails it, so a wrong highest coefficient would."""
    nx, ny = shape
    dx, dy, eta = 2 * np.pi / nx, 1.3 * 2 * np.pi / ny, 0.7
    alpha = t / (2 * (1 / dx**2 + 1 / dy**2))
    bx, by = _faces(nx, ny, dx, dy, "noise", seed=nx + 3 * ny)
    b = eta * ((by - np.roll(by, 1, 1)) / dx - (bx - np.roll(bx, 1, 0)) / dy)
    A, d, eig = _matrix(nx, ny, dx, dy, alpha)
    x = _solve(b, A, eig)
    k, short = _products(b, A, d)
    assert k == {8e-4: 5, 1e-2: 7, 0.02: 8}[t]
    gx, gy = -(np.roll(short, -1, 0) - short) / dy, (np.roll(short, -1, 1) - short) / dx
    assert _curl_error(gx, gy, x, dx, dy) > 16 * EPS * np.abs(x).max()
