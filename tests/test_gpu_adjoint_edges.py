"""Adjoint kernels at the edges of their tiles: narrow, short and odd grids, one strip or block and one more.

The reference is PyTorch autograd through the CPU restatement of the step (dense solves), so the grids stay small
in one direction. Tolerance: the suite's bound for these quantities, 1e-9 relative per field; the FP64 operations
behind a value (a few hundred a cell, a solve to 1e-15) leave five orders of magnitude to it.
"""
import numpy as np
import pytest
import torch

from oracle import torch_step as ts
from tests_helpers import smooth_state

pytestmark = pytest.mark.gpu

REF_TOL = 1e-9


def _rel(got, want):
    floor = max(float(w.abs().max()) for w in want)
    return max(float((g - w).abs().max()) / max(float(w.abs().max()), 1e-3 * floor) for g, w in zip(got, want))


def _ptrs(t):
    return [t[k].data_ptr() for k in range(6)]


def _state(nx, ny, seed):
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    return dx, dy, torch.tensor(np.stack(smooth_state(nx, ny, dx, dy, seed, v_amp=0.3)))


@pytest.mark.parametrize("nx,ny", [(4, 4), (7, 3), (3, 9), (25, 5), (26, 4), (51, 7), (257, 3), (5, 130)])
def test_step_vjp_at_tile_edges(nx, ny):
    import magnetohydrodynamics_simulator_b200 as m

    eta, dt = 3e-2, 1e-3
    dx, dy, U = _state(nx, ny, 3 + nx)
    lam_next = torch.randn(6, ny, nx, generator=torch.Generator().manual_seed(nx * ny), dtype=torch.float64)
    Ut = [U[k].clone().requires_grad_(True) for k in range(6)]
    eta_t = torch.tensor(eta, dtype=torch.float64, requires_grad=True)
    out = ts.imex_step(Ut, dt, eta_t, dx, dy, ts.laplacian_matrix(nx, ny, dx, dy))
    grads = torch.autograd.grad(out, Ut + [eta_t], grad_outputs=list(lam_next))
    adj = m.Adjoint(nx, ny, dx, dy, eta, dt, 1)
    u_d, l_d = U.cuda().contiguous(), lam_next.cuda().contiguous()
    lam = torch.empty_like(u_d)
    geta = adj.step_vjp(_ptrs(u_d), _ptrs(l_d), _ptrs(lam))
    err = _rel(list(lam.cpu()), list(grads[:6]))
    assert err <= REF_TOL, err
    assert abs(geta - float(grads[6])) <= REF_TOL * abs(float(grads[6])), (geta, float(grads[6]))


@pytest.mark.parametrize("nx,ny", [(2, 2), (2, 7), (300, 2), (24, 33), (25, 8), (76, 61), (130, 257)])
def test_rate_vjp_at_tile_edges(nx, ny):
    """The explicit rate alone, also with the result written over its arguments."""
    import magnetohydrodynamics_simulator_b200 as m

    dx, dy, U = _state(nx, ny, 11 + ny)
    w = torch.randn(6, ny, nx, generator=torch.Generator().manual_seed(nx + ny), dtype=torch.float64)
    Ut = [U[k].clone().requires_grad_(True) for k in range(6)]
    want = torch.autograd.grad(ts.explicit_rhs(Ut, dx, dy), Ut, grad_outputs=list(w))
    adj = m.Adjoint(nx, ny, dx, dy, 1e-2, 1e-3, 1)
    u_d, w_d = U.cuda().contiguous(), w.cuda().contiguous()
    out = torch.empty_like(u_d)
    adj.rate_vjp(_ptrs(u_d), _ptrs(w_d), _ptrs(out))
    err = _rel(list(out.cpu()), list(want))
    assert err <= REF_TOL, err
    over_w, over_u = w_d.clone(), u_d.clone()
    adj.rate_vjp(_ptrs(u_d), _ptrs(over_w), _ptrs(over_w))
    adj.rate_vjp(_ptrs(over_u), _ptrs(w_d), _ptrs(over_u))
    assert torch.equal(over_w, out) and torch.equal(over_u, out)
