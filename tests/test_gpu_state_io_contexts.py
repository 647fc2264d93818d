"""State planes in memory of another driver context of the same device: no kernel of this context may touch them, so they
go by the copies, which take them or refuse them, and the context stays usable."""
import numpy as np
import pytest
import torch

from tests_helpers import smooth_state

pytestmark = pytest.mark.gpu


def _ok(r):
    assert int(r[0]) == 0, r[0]
    return r[1] if len(r) == 2 else r[1:]


def test_planes_of_another_context():
    from cuda.bindings import driver as drv

    import magnetohydrodynamics_simulator_b200 as m

    assert torch.cuda.is_available()
    nx, ny = 70, 33
    dx, dy = 2 * np.pi / nx, 2 * np.pi / ny
    u = np.ascontiguousarray(np.stack(smooth_state(nx, ny, dx, dy, 3, v_amp=0.3)))
    plane = nx * ny * 8
    ctx = m.Context(nx, ny, dx, dy, 1e-3)
    host = m.Context(nx, ny, dx, dy, 1e-3)
    host.set_state(list(u))
    _ok(drv.cuInit(0) + (None,))
    dev = _ok(drv.cuDeviceGet(torch.cuda.current_device()))
    other = _ok(drv.cuCtxCreate(0, dev))  # current now
    try:
        src, dst = int(_ok(drv.cuMemAlloc(6 * plane))), int(_ok(drv.cuMemAlloc(6 * plane)))
        _ok(drv.cuMemcpyHtoD(src, u.ctypes.data, 6 * plane) + (None,))
        _ok(drv.cuCtxPopCurrent())
        try:
            ctx.set_state_device([src + k * plane for k in range(6)])
            taken = True
        except m.MHDError:
            taken = False
        if taken:
            assert ctx.cfl_dt() == host.cfl_dt()
            assert np.array_equal(np.stack(ctx.get_state()), u)
            ctx.get_state_device([dst + k * plane for k in range(6)])
            ctx.synchronize()
        ctx.set_state(list(u))
        ctx.step(0.0)
        host.step(0.0)
        for a, b in zip(ctx.get_state(), host.get_state()):
            assert np.array_equal(a, b)
        _ok(drv.cuCtxPushCurrent(other) + (None,))
        if taken:
            back = np.empty_like(u)
            _ok(drv.cuMemcpyDtoH(back.ctypes.data, dst, 6 * plane) + (None,))
            assert np.array_equal(back, u)
    finally:
        drv.cuCtxPushCurrent(other)
        drv.cuCtxDestroy(other)
    ctx.close()
    host.close()
