"""The FP64 fluxes over the range of the numbers (cpp/flux_range.cu): between
equal states they are the physical flux, whatever the scale of density and at
zero pressure too (the flux of either side, which no contact speed enters).
Some thirty roundings of terms no larger than the reference size: 40 units of
2^-53."""
import os
import subprocess

import pytest

from rkdg_heter_calculate_b200 import build

pytestmark = pytest.mark.gpu


def test_fluxes_of_equal_states(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "flux_range")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC,
                    os.path.join(here, "cpp", "flux_range.cu"), build.LIB, "-o", exe,
                    "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(build.LIB)] + build.ARCH, check=True)
    hllc, llf = (float(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert hllc <= 40 * 2.0**-53 and llf <= 40 * 2.0**-53, (hllc, llf)
