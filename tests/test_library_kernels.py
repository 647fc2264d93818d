"""Each solve kernel is in the library once: a copy per translation unit is loaded, and set up, per copy."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

LIB = os.path.join(ROOT, "magnetohydrodynamics_simulator_b200", "libmhd_b200.so")


@pytest.mark.skipif(shutil.which("nm") is None or not os.path.exists(LIB), reason="needs nm and the built library")
@pytest.mark.parametrize("kernel", ["mhd::k_solve(", "mhd::k_cg_cluster(", "mhd::k_cg_band(", "mhd::k_cg_sweep<true>(",
                                    "mhd::k_cg_sweep<false>(", "mhd::k_solve_batch(", "mhd::k_cluster_batch("])
def test_one_copy_of_each_solve_kernel(kernel):
    out = subprocess.run(["nm", "-C", LIB], check=True, capture_output=True, text=True).stdout
    entries = [ln for ln in out.splitlines() if ln.split(maxsplit=2)[1:2] in (["t"], ["T"], ["W"]) and kernel in ln]
    assert len(entries) == 1, entries
