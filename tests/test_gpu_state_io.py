"""Device state in and out of a context and a batch: every value bit for bit, and the CFL step of a state set
through device planes the one of the same state set from the host, whatever memory the planes are."""
import numpy as np
import pytest
import torch

from tests_helpers import smooth_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def m():
    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def _state(nx, ny):
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    return dx, dy, np.stack(smooth_state(nx, ny, dx, dy, nx + ny, v_amp=0.3))


def _planes(u, where):
    """Six planes with u's values: one tensor, separate odd (8-byte aligned) slices, or pinned host memory."""
    if where == "device":
        t = torch.tensor(u, device="cuda")
        return t, [t[k].data_ptr() for k in range(6)]
    if where == "slices":
        t = [torch.cat([torch.zeros(2 * k + 1), torch.tensor(u[k]).flatten(), torch.zeros(3)]).double().cuda()
             for k in range(6)]
        return t, [t[k].data_ptr() + 8 * (2 * k + 1) for k in range(6)]
    t = torch.tensor(u).pin_memory()
    return t, [t[k].data_ptr() for k in range(6)]


@pytest.mark.parametrize("where", ["device", "slices", "pinned"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (255, 3), (257, 5), (3, 700), (640, 411)])
def test_context_state_round_trip(m, nx, ny, where):
    dx, dy, u = _state(nx, ny)
    host = m.Context(nx, ny, dx, dy, 1e-3)
    host.set_state(list(u))
    ctx = m.Context(nx, ny, dx, dy, 1e-3)
    keep, ptrs = _planes(u, where)
    torch.cuda.synchronize()
    ctx.set_state_device(ptrs)
    assert ctx.cfl_dt() == host.cfl_dt()
    out = torch.full((6, ny, nx), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.get_state_device([out[k].data_ptr() for k in range(6)])
    ctx.synchronize()
    assert np.array_equal(out.cpu().numpy(), u)
    back, bptrs = _planes(np.zeros_like(u), where)
    torch.cuda.synchronize()
    ctx.get_state_device(bptrs)
    ctx.synchronize()
    for k in range(6):
        got = back[k].flatten()[2 * k + 1:-3].reshape(ny, nx) if where == "slices" else back[k]
        assert np.array_equal(got.cpu().numpy(), u[k])
        if where == "slices":
            assert not back[k][:2 * k + 1].any() and not back[k][-3:].any()


def test_state_from_its_own_planes(m):
    nx, ny = 130, 37
    dx, dy, u = _state(nx, ny)
    ctx = m.Context(nx, ny, dx, dy, 1e-3)
    ctx.set_state(list(u))
    dt = ctx.cfl_dt()
    ctx.set_state_device(ctx.state_device_pointers())
    assert ctx.cfl_dt() == dt
    assert np.array_equal(np.stack(ctx.get_state()), u)


@pytest.mark.parametrize("where", ["device", "slices", "pinned"])
def test_batch_state_round_trip(m, where):
    sizes = [(5, 4), (64, 64), (300, 9)]
    states = [_state(nx, ny) for nx, ny in sizes]
    spec = [{"nx": nx, "ny": ny, "dx": s[0], "dy": s[1], "eta": 1e-3} for (nx, ny), s in zip(sizes, states)]
    b, host = m.Batch(spec), m.Batch(spec)
    for i, (dx, dy, u) in enumerate(states):
        keep, ptrs = _planes(u, where)
        torch.cuda.synchronize()
        b.set_state_device(i, ptrs)
        host.set_state(i, list(u))
        assert b.cfl_dt(i) == host.cfl_dt(i)
    for i, (dx, dy, u) in enumerate(states):
        out = torch.zeros(u.shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        b.get_state_device(i, [out[k].data_ptr() for k in range(6)])
        b.synchronize()
        assert np.array_equal(out.cpu().numpy(), u)
