"""The FP64 reciprocal and roots of the flux arithmetic (csrc/roots.cuh)
against CUDA's IEEE divide and square root.  Each refined value is within one
unit in the last place of the exact one, as the IEEE value is within half of
one, so the two differ by at most one; the reciprocal root, checked through
its product with the root, by at most three (its own unit, the root's half
and the product's half, in units of 2^-52)."""
import os
import subprocess

import pytest

from rkdg_heter_calculate_b200 import build

pytestmark = pytest.mark.gpu


def test_roots_are_within_one_ulp(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "roots")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-I", build.CSRC, os.path.join(here, "cpp", "roots.cu"),
                    "-o", exe] + build.ARCH, check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    rcp, rcp_neg, root, inv_root, at_zero, below = (int(v) for v in out)
    assert rcp <= 1 and rcp_neg <= 1 and root <= 1 and inv_root <= 3, out
    assert at_zero == 1 and below == 1, out
