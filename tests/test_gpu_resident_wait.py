"""What a resident solve does when data that a tile waits for never arrives
(csrc/resident.cuh): the wait gives up after two seconds and the launch reports
it, whichever stage it was and whatever arrives later (cpp/resident_wait.cu)."""
import os
import subprocess

import pytest

from rkdg_heter_calculate_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    """(error word, done, steps, ms) after each of two queued launches, and
    (refused, last error) of one too large for the device."""
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path_factory.mktemp("wait") / "resident_wait")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC,
                    os.path.join(here, "cpp", "resident_wait.cu"), build.LIB, "-o", exe,
                    "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(build.LIB)] + build.ARCH, check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


def test_a_lost_mean_is_reported(launches):
    error, _, _, ms = launches[0]
    assert error == 2 and 1500 < ms < 10000, launches


def test_launches_behind_a_lost_wait_leave_at_once(launches):
    """A whole advance is queued without a read-back in between: none of the
    launches behind the failed one may wait again, or step on from its state."""
    (_, done, steps, _), (error, _, steps2, ms) = launches[:2]
    assert done == 1 and steps == steps2 == 0 and error == 2 and ms < 500, launches


def test_a_launch_too_large_is_refused_without_an_error(launches):
    """The caller falls back to the stage kernels."""
    assert launches[2] == (1, 0)
