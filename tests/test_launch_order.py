"""What the kernels that overlap their predecessor must do, read from their
source: they are launched with programmatic stream serialization
(launch_dependent), so nothing but griddepcontrol.wait orders them after the
launch ahead, and a run that goes well does not show that a wait is missing."""
import os
import re

import pytest

from rkdg_heter_calculate_b200 import build

SOURCES = ["kernels.cu", "device.cuh", "stage_tiled.cuh", "stage_fp64.cuh"]


def source(name):
    text = open(os.path.join(build.CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def body(text, at):
    """The braced block that starts at or after position at."""
    start = i = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def overlapping_kernels():
    """name -> body of the kernels launched early."""
    text = "\n".join(source(f) for f in SOURCES)
    launched = set(re.findall(r"launch_dependent\([^,]+,\s*(\w+)", source("kernels.cu")))
    launched.discard("void")  # the launcher's own definition
    launched.discard("kernel")  # stage_kernel(): the two below
    launched |= {"tiled_stage_kernel", "stage_fp64_kernel"}
    out = {}
    for name in launched:
        m = re.search(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s*)?" + name + r"\(", text)
        assert m, name
        out[name] = body(text, m.end())
    return out


def test_overlapping_kernels_are_found():
    assert set(overlapping_kernels()) == {"step_begin_kernel", "tiled_limiter_kernel", "tiled_stage_kernel",
                                          "stage_fp64_kernel"}


@pytest.mark.parametrize("name", sorted(overlapping_kernels()))
def test_no_path_leaves_before_the_wait(name):
    """A launch whose blocks all leave without waiting (a tile list that is
    empty) completes before the launch ahead of it, and the next launch, which
    waits for it alone, then runs beside that one."""
    text = overlapping_kernels()[name]
    assert "grid_dependency_wait()" in text
    for m in re.finditer(r"\breturn\b", text):
        assert "grid_dependency_wait()" in text[: m.start()], text[max(0, m.start() - 80): m.end()]


# arguments of __ldg: the tables of a mesh, a rule or a solve, which no kernel writes
TABLES = ("ta.", "&ta.", "jinv2 ", "j2 ", "conn ", "lim ", "&g[", "t)", "t +")


def test_written_memory_is_not_read_through_the_read_only_path():
    """A kernel that starts early is alive while the one ahead writes the
    states and control blocks; the read-only path is for memory that nothing
    writes in the kernel's lifetime, and its loads may move above the wait."""
    for name in ["kernels.cu", "device.cuh", "stage_tiled.cuh", "stage_fp64.cuh"]:
        for m in re.finditer(r"__ldg\(([^;]*)", source(name)):
            assert m.group(1).startswith(TABLES), (name, m.group(0)[:60])
    limiter = re.search(r"tiled_limiter_kernel\(.*?\{", source("kernels.cu"), re.S).group(0)
    for p in limiter.split(","):
        if re.search(r"\b(U|ctl)$", p.strip()):
            assert "__restrict__" not in p, p
