import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


def pytest_collection_modifyitems(config, items):
    """The tests that compare with programs built from the reference's own sources fail where those are not at hand
    (oracle/_ref is not built): they run last then, so that a run that stops at the first failure has run the others."""
    built = ("libmhdref.so", "integrator_main_ref", "integrator_main_b200")
    if all(os.path.exists(os.path.join(ROOT, "oracle", "_ref", f)) for f in built):
        return
    needs = ("test_gpu_dropin.py", "test_gpu_headline_parity.py")
    items.sort(key=lambda it: os.path.basename(str(it.fspath)) in needs)


def load_golden(name):
    return dict(np.load(os.path.join(GOLDEN, name)))


def fields(d, prefix):
    return [d[f"{prefix}_{n}"] for n in ("rho", "mx", "my", "E", "bxf", "byf")]


@pytest.fixture(scope="session")
def oracle_built():
    from oracle import oracle

    oracle.oracle_lib()
    return oracle


def gpu_available():
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False
