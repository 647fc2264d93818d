"""The autotuner chooses a decomposition of the ordinary CG iterations only where an instance takes them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def m():
    import torch

    assert torch.cuda.is_available()
    import magnetohydrodynamics_simulator_b200 as mod

    return mod


def _tuned(m, sizes, etas):
    b = m.Batch([{"nx": nx, "ny": ny, "dx": 2 * np.pi / nx, "dy": 2 * np.pi / ny, "eta": eta}
                 for (nx, ny), eta in zip(sizes, etas)])
    for i, (nx, ny) in enumerate(sizes):
        b.set_state(i, m.problems.orszag_tang(nx, ny, 2 * np.pi / nx, 2 * np.pi / ny))
    b.set_tuning(40, 96, 1)  # 96 is no candidate
    t = b.autotune()
    b.step()
    assert b.synchronize_status()[0] == 0
    b.close()
    return t


@pytest.mark.parametrize("sizes,etas", [([(64, 64), (48, 60)], [1e-3, 1e-2]),             # clusters
                                        ([(300, 290), (64, 64), (400, 250)], [1e-4, 1e-3, 5e-4])])  # and two passes
def test_solver_setting_stays_where_nothing_uses_it(m, sizes, etas):
    t = _tuned(m, sizes, etas)
    assert (t["cg_rows"], t["cg_order"]) == (96, 1)
    assert t["stage_ms"] > 0 and t["cg_ms"] > 0


def test_solver_setting_is_chosen_where_an_instance_uses_it(m):
    t = _tuned(m, [(300, 290), (64, 64)], [0.5, 1e-3])
    assert t["cg_rows"] != 96
