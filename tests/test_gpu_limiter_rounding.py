"""The reciprocals and roots that decide whether an FP32 element is limited
round as IEEE does (csrc/device.cuh, cpp/limiter_rounding.cu)."""
import os
import subprocess

import pytest

from rkdg_heter_calculate_b200 import build

pytestmark = pytest.mark.gpu


def test_limiter_rounds_as_ieee(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "rounding")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC,
                    os.path.join(here, "cpp", "limiter_rounding.cu"), build.LIB, "-o", exe,
                    "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(build.LIB)] + build.ARCH, check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["0", "0", "0"]
