"""Kernel attributes and what a device answers about them are kept per device
(csrc/per_device.hpp): a process may drive several."""
import glob
import os
import re
import subprocess

from rkdg_heter_calculate_b200 import build


def test_each_device_has_its_own_value(tmp_path):
    exe = str(tmp_path / "per_device")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", build.CSRC, os.path.join(here, "cpp", "per_device.cpp"),
                    "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["10", "11", "1", "1"]


def test_no_device_state_is_kept_per_process_or_thread():
    """Variables of the CUDA sources' host code that outlive a call."""
    for path in glob.glob(os.path.join(build.CSRC, "*.cu")) + glob.glob(os.path.join(build.CSRC, "*.cuh")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        assert "thread_local" not in text and "once_flag" not in text, path
        for m in re.finditer(r"\bstatic\s+(?!constexpr|__|inline)([\w:<>, ]+?)\s+(\w+)\s*(=|;|\{)", text):
            assert m.group(1).startswith("PerDevice<"), (path, m.group(0))
